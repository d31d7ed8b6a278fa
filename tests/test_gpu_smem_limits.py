"""Shared-memory limits of kernels whose tiles or bins vary from call to call.

The limit that a launch is held to belongs to the kernel, not to the handle: it
must cover every size a call may ask for, whichever thread asked last, and the
sizes whose dynamic part alone just fills the default 48 KB.
"""
from __future__ import annotations

import re
import threading

import numpy as np
import pytest

from helpers import L, random_state

pytestmark = pytest.mark.gpu


def lattice(engine, shape=(16, 16, 16), **kw):
    kw = dict(dict(nfld=1, length=8.0, laplacian=L.LAP_FD27, precision=L.FP64, model=L.MODEL_PHI4,
                   model_params=(1.0,)), **kw)
    g = engine.Lattice(L.make_config(shape, **kw))
    nx, ny, nz = shape
    g.set_state(*random_state((kw["nfld"], nz, ny, nx), seed=2, mean=0.5))
    return g


@pytest.mark.parametrize("nb", [192, 383, 384, 385, 767, 768, 769, 1536, 2048])
@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
def test_bin_counts(engine, nb, prec):
    """Eight warps' bins of one, two or four sums fill 48 KB at 768, 384 and 192 bins; more bins than that
    hold the same sums."""
    g = lattice(engine, precision=prec, model=L.MODEL_DOUBLE_WELL, model_params=(0.01,), gw=True, gw_coupling=1.0)
    u = np.random.default_rng(1).standard_normal((2, 6, 16, 16, 16))
    g.set_gw_state(u[0], u[1])
    calls = [lambda n: g.spectrum(L.SPEC_FLD, 0, L.SPEC_WEIGHTED, n), lambda n: g.spectrum_bin(L.SPEC_FLD, 0, n),
             lambda n: g.crossspec_3d(L.SPEC_FLDP, 0, L.SPEC_FLD, 0, n), g.gw_spectrum]
    for call in calls:
        few, many = call(20), call(nb)
        for a, b in zip(few, many):
            assert len(b) == nb and np.allclose(b[:20], a, rtol=1e-13, atol=1e-13 * np.max(np.abs(a)))


def in_threads(*jobs):
    bad = []

    def go(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001 (reported below)
            bad.append(e)
    ts = [threading.Thread(target=go, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[0]


def test_bins_in_two_threads(engine):
    g, h = lattice(engine), lattice(engine)

    def many():
        for _ in range(1500):
            g.spectrum(L.SPEC_FLD, 0, L.SPEC_WEIGHTED, 2048)

    def fewer():
        for _ in range(1500):
            h.spectrum(L.SPEC_FLD, 0, L.SPEC_WEIGHTED, 400)
    in_threads(many, fewer)


def test_stencil_tiles_in_two_threads(engine, tmp_path, monkeypatch):
    """Two lattices of one kernel whose tiles have eight and four rows (57 and 34 KB)."""
    monkeypatch.setenv("LAT_NO_GRAPHS", "1")  # launches, not replays
    kw = dict(model=L.MODEL_DOUBLE_WELL, model_params=(0.01,), gw=True, gw_coupling=1.0)
    cache = tmp_path / "tune.jsonl"
    first = lattice(engine, **kw)
    first.autotune(cache)
    line = cache.read_text()
    gs = []
    for ty in (8, 4):
        c = tmp_path / ("tune%d.jsonl" % ty)
        c.write_text(re.sub(r'"ty": \d+', '"ty": %d' % ty, line))
        gs.append(lattice(engine, **kw))
        gs[-1].autotune(c)
        assert gs[-1].tuning()[1] == ty

    def steps(g):
        for _ in range(20):
            g.symp(2, 1e-3, 200)
            g.sync()
    in_threads(lambda: steps(gs[0]), lambda: steps(gs[1]))
    a, b = gs[0].get_state()[0], gs[1].get_state()[0]
    assert np.max(np.abs(a - b)) <= 1e-9
