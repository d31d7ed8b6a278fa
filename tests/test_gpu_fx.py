"""FP64 spectral lattices on the fixed-point passes (csrc/k_fx.cuh), which AUTO
takes where they tile the sides, against the cuFFT path on identical inputs.

Both evaluate laplacian_3d (Pseudospec/openmp_dev/fftw_mod.f90:177-207) to FP64
rounding; the tolerances are those of the other FP64 path comparison: 1e-12 of
the fields, ten times that of the momenta.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err
from helpers import L, random_state

pytestmark = pytest.mark.gpu

# every line length along every axis, the smallest tiles (16 x-columns with two fields,
# 32 with one), sides that differ
CASES = [((16, 16, 16), 2), ((32, 512, 16), 2), ((16, 32, 512), 2), ((512, 16, 32), 2), ((32, 32, 32), 2),
         ((64, 64, 64), 1), ((512, 64, 32), 1), ((128, 512, 16), 1), ((128, 16, 512), 1), ((256, 128, 64), 1)]


# sides that run padded (k_fxg.cuh): both edges of every padded length (9..32 on 64 points,
# 33..64, 65..128, 129..256), odd numbers of lines with one field, padded beside direct sides
CASES += [((9, 32, 33), 2), ((64, 65, 20), 2), ((17, 129, 12), 2), ((256, 9, 30), 2), ((48, 36, 255), 2),
          ((65, 39, 13), 1), ((128, 33, 15), 1), ((150, 96, 10), 1), ((64, 18, 128), 1)]


def pair(engine, shape, nf, **kw):
    out = []
    for impl in (L.SPEC_IMPL_AUTO, L.SPEC_IMPL_CUFFT):
        c = L.make_config(shape, nfld=nf, length=0.25 * shape[0], laplacian=L.LAP_SPECTRAL, precision=L.FP64,
                          spectral_impl=impl, **kw)
        out.append(engine.Lattice(c))
    assert out[0].tuning()[5] == L.SPEC_IMPL_SEPARABLE and out[1].tuning()[5] == L.SPEC_IMPL_CUFFT
    return out


@pytest.mark.parametrize("conf", [False, True])
@pytest.mark.parametrize("shape,nf", CASES)
def test_fixed_point_passes_match_cufft(engine, shape, nf, conf):
    a, b = pair(engine, shape, nf, background=L.BG_CONFORMAL if conf else L.BG_MINKOWSKI,
                model=L.MODEL_PHI4_G2 if nf == 2 else L.MODEL_PHI4,
                model_params=(1.0, 2.0) if nf == 2 else (1.0,))
    f, p = random_state((nf, shape[2], shape[1], shape[0]), seed=11, mean=1.0, amp=0.05)
    for g in (a, b):
        g.set_state(f, p)
        if conf:
            g.set_scale_factor(1.0, 0.0)
            g.calc_metric()
        g.symp(4, 0.01, 3)
    (fa, pa), (fb, pb) = a.get_state(), b.get_state()
    assert rel_err(fa, fb) <= 1e-12 and rel_err(pa, pb) <= 1e-11
    if conf:
        (aa, apa), (ab, apb) = a.scale_factor(), b.scale_factor()
        assert abs(aa - ab) <= 1e-12 * ab and abs(apa - apb) <= 1e-11 * abs(apb)


@pytest.mark.parametrize("model,params,nf", [(L.MODEL_PHI4, (0.7,), 2), (L.MODEL_DOUBLE_WELL, (0.01,), 1),
                                             (L.MODEL_DOUBLE_WELL, (0.01,), 2), (L.MODEL_FREE, (1.3,), 1),
                                             (L.MODEL_FREE, (1.3,), 2)])
def test_models(engine, model, params, nf):
    shape = (64, 32, 16) if nf == 2 else (64, 64, 32)
    a, b = pair(engine, shape, nf, background=L.BG_CONFORMAL, model=model, model_params=params)
    f, p = random_state((nf, shape[2], shape[1], shape[0]), seed=4, mean=0.5, amp=0.1)
    for g in (a, b):
        g.set_state(f, p)
        g.set_scale_factor(1.0, -0.5)
        g.symp(2, 0.01, 5)
    assert rel_err(a.get_state()[0], b.get_state()[0]) <= 1e-12
    assert abs(a.scale_factor()[1] - b.scale_factor()[1]) <= 1e-11 * abs(b.scale_factor()[1])


def test_uneven_and_vanishing_fields(engine):
    """A field that is zero stays exactly zero beside one that fluctuates, a field 1e-9 times the
    other keeps its own accuracy, and infinities reach no other line than their own."""
    shape, n = (64, 64, 64), 64 ** 3
    a, b = pair(engine, shape, 2, model=L.MODEL_FREE, model_params=(1.0,))
    f, p = random_state((2, 64, 64, 64), seed=9, mean=0.0, amp=0.1)
    f[1], p[1] = 0.0, 0.0
    for g in (a, b):
        g.set_state(f, p)
        g.symp(4, 0.01, 2)
    assert np.all(a.get_state()[0][1] == 0.0) and np.all(a.get_state()[1][1] == 0.0)
    f2, p2 = random_state((2, 64, 64, 64), seed=10, mean=0.0, amp=0.1)
    f2[1] *= 1e-9
    p2[1] *= 1e-9
    for g in (a, b):
        g.set_state(f2, p2)
        g.symp(4, 0.01, 2)
    for l in range(2):
        assert rel_err(a.get_state()[0][l], b.get_state()[0][l]) <= 1e-12
    f2[0, 5, 6, 7] = np.inf
    a.set_state(f2, p2)
    a.symp(2, 0.01, 1)  # one kick: the site's own x, y and z lines
    bad = ~np.isfinite(a.get_state()[1][0])
    line = np.zeros((64, 64, 64), bool)
    line[5, 6, :] = line[5, :, 7] = line[:, 6, 7] = True
    assert np.array_equal(bad, line) and np.all(np.isfinite(a.get_state()[1][1]))
    a.sync()  # a static background reports non-finite fields with the energies, as on cuFFT
    with pytest.raises(engine.LatticeError) as e:
        a.energies()
    assert e.value.code == 4


def test_evolution_is_reproducible(engine):
    out = []
    for _ in range(2):
        a, _ = pair(engine, (64, 64, 64), 2, background=L.BG_CONFORMAL, model=L.MODEL_PHI4_G2, model_params=(1.0, 2.0))
        a.init_vacuum(3, [1.0, 0.0], [0.0, 0.0], [3.0, 2.0], amp=1e-6)
        a.set_scale_factor(1.0, 0.0)
        a.calc_metric()
        a.symp(4, 0.01, 4)
        out.append((*a.get_state(), a.scale_factor()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1]) and out[0][2] == out[1][2]


@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
@pytest.mark.parametrize("shape", [(16, 16, 16), (16, 512, 32), (512, 32, 16), (32, 16, 512), (64, 128, 256)])
def test_spectrum_transform_matches_numpy(engine, shape, prec):
    """The fixed-point real-to-complex transform under the spectra (csrc/k_fxr.cuh), every line
    length along every axis, against numpy's FP64 transform of the same numbers binned like
    spectrum_bin; each bin is a sum of squares, so FP64 rounding leaves it within 1e-11."""
    nx, ny, nz = shape
    c = L.make_config(shape, nfld=1, length=1.0 * nx, laplacian=L.LAP_FD7, precision=prec)
    g = engine.Lattice(c)
    f, p = random_state((1, nz, ny, nx), seed=21, mean=3.0, amp=1e-3)
    g.set_state(f, p)
    x, y = g.get_state()  # what the handle holds (FP32-Kahan: phi_hi - c)
    nb = g.nbins()
    fold = [np.minimum(np.arange(n), n - np.arange(n)) for n in (nz, ny)] + [np.arange(nx // 2 + 1)]
    m2 = fold[0][:, None, None] ** 2 + fold[1][None, :, None] ** 2 + fold[2][None, None, :] ** 2
    l = np.floor(np.sqrt(m2)).astype(int).ravel()
    w = np.broadcast_to(np.where((fold[2] == 0) | (2 * fold[2] == nx), 1.0, 2.0), m2.shape).ravel()
    for what, a in ((L.SPEC_FLD, x[0]), (L.SPEC_FLDP, y[0])):
        F = np.fft.rfftn(a)
        S = np.bincount(l, w * (F.real ** 2 + F.imag ** 2).ravel(), nb)[:nb]
        W = np.bincount(l, w, nb)[:nb]
        got, cnt = g.spectrum_bin(what, 0, nb)
        assert np.array_equal(cnt, W)
        ok = W > 0
        assert np.max(np.abs(got[ok] * W[ok] / S[ok] - 1)) <= 1e-11
