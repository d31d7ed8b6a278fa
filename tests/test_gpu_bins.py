"""Shell binning (csrc/k_bin.cu) against numpy: odd and even sides, rows shorter
and longer than a warp, one bin and the most there are (one warp a block), power,
counts, cross spectra and the TT projection.

Every bin is a sum of FP64 products of the same transform to rounding, so bins
agree to 1e-11 of the bin's absolute sum; counts are exact.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import L, random_state

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (15, 9, 21), (66, 34, 10), (33, 64, 31), (20, 18, 130)]


def shells(shape):
    nx, ny, nz = shape
    k = [np.arange(nx // 2 + 1), np.minimum(np.arange(ny), ny - np.arange(ny)),
         np.minimum(np.arange(nz), nz - np.arange(nz))]
    m2 = (k[2][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[0][None, None, :] ** 2).ravel()
    l = np.floor(np.sqrt(m2)).astype(int)
    w = np.broadcast_to(np.where((k[0] == 0) | (2 * k[0] == nx), 1.0, 2.0), (nz, ny, nx // 2 + 1)).ravel()
    p = np.sqrt(m2.astype(float))
    return l, w, (1 - (l - p) ** 2) ** 2, (1 - (l + 1 - p) ** 2) ** 2


def two_bin(shape, v, nb):
    l, w, c0, c1 = shells(shape)
    n = max(nb, l.max() + 2)
    a, b = np.bincount(l, w * c0 * v, n), np.bincount(l, w * c1 * v, n)
    a[1:] += b[:-1]
    return a[:nb]


@pytest.mark.parametrize("nb", [1, 7, 2048])
@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
@pytest.mark.parametrize("shape", SHAPES)
def test_power_and_cross(engine, shape, prec, nb):
    nx, ny, nz = shape
    g = engine.Lattice(L.make_config(shape, nfld=2, length=1.0, laplacian=L.LAP_SPECTRAL, precision=prec,
                                     model=L.MODEL_PHI4_G2, model_params=(1.0, 2.0)))
    g.set_state(*random_state((2, nz, ny, nx), seed=5, mean=0.3, amp=1.0))
    f, p = g.get_state()
    F, G = np.fft.rfftn(f[0]).ravel(), np.fft.rfftn(p[0]).ravel()
    pw = np.abs(F) ** 2
    W = two_bin(shape, np.ones(F.size), nb)
    ok = W != 0
    S, Wg = g.spectrum(L.SPEC_FLD, 0, L.SPEC_WEIGHTED, nb)
    assert np.allclose(Wg, W, rtol=1e-12, atol=0)
    assert np.allclose(S[ok] * W[ok], two_bin(shape, pw, nb)[ok], rtol=1e-11, atol=0) and np.all(S[~ok] == 0)
    l, w, _, _ = shells(shape)
    n = max(nb, l.max() + 1)
    cnt = np.bincount(l, w, n)[:nb]
    S, Wg = g.spectrum_bin(L.SPEC_FLD, 0, nb)
    assert np.array_equal(Wg, cnt)
    assert np.allclose(S * np.maximum(cnt, 1), np.bincount(l, w * pw, n)[:nb], rtol=1e-11, atol=0)
    if prec == L.FP32_KAHAN and nx * ny * nz % 2:
        return  # the second FP64 copy starts off cuFFT's 16-byte alignment: refused with its error
    x = G * F.conj()
    re, im = g.crossspec_3d(L.SPEC_FLDP, 0, L.SPEC_FLD, 0, nb)
    size = two_bin(shape, np.abs(x), nb)
    for got, v in ((re, x.real), (im, x.imag)):
        assert np.all(np.abs(got[ok] * W[ok] - two_bin(shape, v, nb)[ok]) <= 1e-11 * size[ok])


@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
@pytest.mark.parametrize("shape", SHAPES[1:])
def test_tt_projection(engine, shape, prec):
    nx, ny, nz = shape
    g = engine.Lattice(L.make_config(shape, nfld=1, length=1.0 * nx, laplacian=L.LAP_FD27, precision=prec,
                                     model=L.MODEL_DOUBLE_WELL, model_params=(0.01,), gw=True, gw_coupling=2.0))
    rng = np.random.default_rng(8)
    u = rng.standard_normal((2, 6, nz, ny, nx))
    g.set_gw_state(u[0], u[1])
    pu = g.gw_state()[1]
    F = [np.fft.rfftn(v) for v in pu]
    at = ((0, 3, 4), (3, 1, 5), (4, 5, 2))
    s = [np.sin(2 * np.pi * np.arange(m) / n) for m, n in ((nx // 2 + 1, nx), (ny, ny), (nz, nz))]
    k = [s[0][None, None, :] + 0 * F[0].real, s[1][None, :, None] + 0 * F[0].real, s[2][:, None, None] + 0 * F[0].real]
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    inv = np.where(k2 > 0, 1 / np.where(k2 > 0, k2, 1), 0)
    P = [[(i == j) - k[i] * k[j] * inv for j in range(3)] for i in range(3)]
    A = [[sum(P[i][m] * F[at[m][j]] for m in range(3)) for j in range(3)] for i in range(3)]
    tr = A[0][0] + A[1][1] + A[2][2]
    tot = sum(np.abs(sum(A[i][m] * P[m][j] for m in range(3)) - 0.5 * P[i][j] * tr) ** 2
              for i in range(3) for j in range(3)) * (k2 > 0)
    # modes whose lattice momentum is only the rounding of sin(pi) have no defined direction
    tiny = (k2 < 1e-24) & (k2 > 0)
    l, w, _, _ = shells(shape)
    nb = 40
    n = max(nb, l.max() + 1)
    S, W = g.gw_spectrum(nb)
    cnt = np.bincount(l, w, n)[:nb]
    assert np.array_equal(W, cnt)
    ref, loose = np.bincount(l, w * tot.ravel(), n)[:nb], np.bincount(l, tiny.ravel(), n)[:nb] > 0
    tol = 1e-11 if prec == L.FP64 else 2e-5  # FP32 transform of FP32 momenta
    ok = (cnt > 0) & ~loose
    assert np.all(np.abs(S[ok] * cnt[ok] - ref[ok]) <= tol * ref[ok])
