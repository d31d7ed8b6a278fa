"""Energies of one state do not depend on the launch shapes that autotuning found for other passes."""
from __future__ import annotations

import re

import numpy as np
import pytest

from helpers import L, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
@pytest.mark.parametrize("lap,shape", [(L.LAP_SPECTRAL, (128, 64, 64)), (L.LAP_SPECTRAL, (60, 50, 45)),
                                       (L.LAP_FD7, (96, 64, 64)), (L.LAP_FD27, (72, 66, 60))])
def test_energies_of_tuned_handles(engine, tmp_path, lap, shape, prec):
    nx, ny, nz = shape
    cfg = L.make_config(shape, nfld=1, length=8.0, laplacian=lap, precision=prec, model=L.MODEL_PHI4,
                        model_params=(1.0,))
    state = random_state((1, nz, ny, nx), seed=4, mean=0.5)
    g = engine.Lattice(cfg)
    g.set_state(*state)
    e = [g.energies()]
    g.autotune(tmp_path / "t.jsonl")
    line = (tmp_path / "t.jsonl").read_text()
    for bps in (1, 8):
        c = tmp_path / ("t%d.jsonl" % bps)
        c.write_text(re.sub(r'"pw_bps": \d+', '"pw_bps": %d' % bps, line))
        h = engine.Lattice(cfg)
        h.set_state(*state)
        h.autotune(c)
        assert h.tuning()[4] == bps
        e.append(h.energies())
    assert np.array_equal(e[0], e[1]) and np.array_equal(e[0], e[2])  # the same sums, in the same order
