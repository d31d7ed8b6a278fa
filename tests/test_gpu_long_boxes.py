"""Long thin and wide boxes: shapes whose longest side is far beyond the others.

Spectra of sides beyond 4096 points, which hold |n|^2 past the last shell (2047),
against numpy; stencil steps and energies of more rows or planes than a grid of four
rows a block holds, against the same leapfrog in numpy.  Counts and weights hold no data: they agree to rounding.  A bin's
modes carry the rounding of an FP64 transform, below 1e-11 of the mean power.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import L, random_state

pytestmark = pytest.mark.gpu


def folded(n, half=False):
    i = np.arange(n // 2 + 1) if half else np.arange(n)
    return np.minimum(i, n - i).astype(np.int64)


@pytest.mark.parametrize("nb", [100, 2048])
@pytest.mark.parametrize("shape", [(8200, 4, 2), (2, 8201, 4), (4, 2, 9000), (131072, 2, 2), (2, 2, 131072)])
def test_spectra(engine, shape, nb):
    nx, ny, nz = shape
    g = engine.Lattice(L.make_config(shape, nfld=1, length=1.0, laplacian=L.LAP_FD7, precision=L.FP64,
                                     model=L.MODEL_PHI4, model_params=(1.0,)))
    g.set_state(*random_state((1, nz, ny, nx), seed=3, mean=0.2, amp=1.0))
    F = np.abs(np.fft.rfftn(g.get_state()[0][0])).ravel() ** 2
    kx, ky, kz = folded(nx, True), folded(ny), folded(nz)
    m2 = (kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2).ravel()
    w = np.broadcast_to(np.where((kx == 0) | (2 * kx == nx), 1.0, 2.0), (nz, ny, nx // 2 + 1)).ravel()
    p = np.sqrt(m2.astype(float))
    l = np.floor(p).astype(np.int64)
    keep = l < nb
    l, w, p, F, tot = l[keep], w[keep], p[keep], F[keep], F.mean()
    c = [(1 - (l - p) ** 2) ** 2, (1 - (l + 1 - p) ** 2) ** 2]

    def two_bin(v):
        out = np.bincount(l, w * c[0] * v, nb + 1)
        out[1:] += np.bincount(l, w * c[1] * v, nb + 1)[:-1]
        return out[:nb]

    one = np.ones_like(F)
    W, cnt = two_bin(one), np.bincount(l, w, nb)
    S, Wg = g.spectrum(L.SPEC_FLD, 0, L.SPEC_WEIGHTED, nb)
    assert np.allclose(Wg, W, rtol=1e-12, atol=0)
    assert np.all(np.abs(S * np.where(W != 0, W, 1) - two_bin(F)) <= 1e-11 * (two_bin(F) + tot * W))
    S, Wg = g.spectrum_bin(L.SPEC_FLD, 0, nb)
    assert np.array_equal(Wg, cnt)
    assert np.all(np.abs(S * np.maximum(cnt, 1) - np.bincount(l, w * F, nb)) <= 1e-11 * (np.bincount(l, w * F, nb) + tot * cnt))
    g.close()


@pytest.mark.parametrize("mode", [L.SPEC_WEIGHTED, L.SPEC_COUNT])
@pytest.mark.parametrize("shape", [(8200, 4, 2), (131072, 2, 2), (2, 131072, 2), (2, 2, 131072)])
def test_noalloc_spectra(engine, shape, mode):
    """The allocation-free binning of the same transform: sums in another order."""
    torch = pytest.importorskip("torch")
    nx, ny, nz = shape
    nb = 300
    g = engine.Lattice(L.make_config(shape, nfld=1, length=1.0, laplacian=L.LAP_FD7, precision=L.FP64,
                                     model=L.MODEL_PHI4, model_params=(1.0,)))
    f, p = random_state((1, nz, ny, nx), seed=3, mean=0.2, amp=1.0)
    g.set_state(f, p)
    S, W = g.spectrum(L.SPEC_FLD, 0, mode, nb)
    F = torch.from_numpy(np.fft.rfftn(f[0])).cuda().contiguous()
    out = torch.zeros(2 * nb, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert engine._lib.lat_spectrum_noalloc(F.data_ptr(), nx, ny, nz, L.FP64, mode, nb, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.allclose(got[nb:], W, rtol=1e-12, atol=0)
    assert np.all(np.abs(got[:nb] - S) <= 1e-11 * (S + np.mean(S)))
    g.close()


@pytest.mark.parametrize("prec,tol", [(L.FP64, 1e-12), (L.FP32_KAHAN, 1e-5)])
@pytest.mark.parametrize("shape", [(131072, 2, 2), (2, 131072, 2), (2, 2, 131072)])
def test_spectral_laplacian(engine, shape, prec, tol):
    """Squares of mode numbers beyond 32 bits: read-out, gradient energy and one kick of a long spectral box.
    The largest mode number is 65536; a transform's rounding is relative to the largest derivative."""
    nx, ny, nz = shape
    g = engine.Lattice(L.make_config(shape, nfld=1, length=1.0 * nx, laplacian=L.LAP_SPECTRAL, precision=prec,
                                     model=L.MODEL_FREE, model_params=(0.0,)))
    g.set_state(*random_state((1, nz, ny, nx), seed=5, mean=0.0, amp=1.0))
    f, p = (v[0] for v in g.get_state())
    k = [np.fft.fftfreq(n, 1.0 / n) * 2 * np.pi / n for n in (nz, ny, nx)]  # dx = 1
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    F = np.fft.fftn(f)
    ref = np.fft.ifftn(-k2 * F).real
    top = np.max(np.abs(ref))
    assert np.max(np.abs(g.laplacian() - ref)) <= tol * top
    want = 0.5 * np.sum(k2 * np.abs(F) ** 2) / float(f.size) ** 2
    assert abs(g.energies()[L.E_GE_LAP] - want) <= tol * want
    dt = 0.01
    g.symp(2, dt, 1)
    f = f + 0.5 * dt * p
    p = p + dt * np.fft.ifftn(-k2 * np.fft.fftn(f)).real
    f = f + 0.5 * dt * p
    got = g.get_state()
    assert np.max(np.abs(got[1][0] - p)) <= tol * top and np.max(np.abs(got[0][0] - f)) <= tol * top
    g.close()


def neighbours(g, lap):
    """Sums over the 6 face and, with 27 points, 12 edge and 8 corner neighbours."""
    n = lambda v, d: np.roll(v, 1, d) + np.roll(v, -1, d)  # noqa: E731
    sx, sy = n(g, 2), n(g, 1)
    r = [sx + sy + n(g, 0)]
    if lap == L.LAP_FD27:
        sxy = n(sx, 1)
        r += [sxy + n(sx + sy, 0), n(sxy, 0)]
    return r


@pytest.mark.parametrize("prec,tol", [(L.FP64, 1e-12), (L.FP32_KAHAN, 2e-5)])
@pytest.mark.parametrize("shape,lap", [((2, 262200, 2), L.LAP_FD7), ((2, 262200, 2), L.LAP_FD27),
                                       ((3, 2, 140000), L.LAP_FD7), ((3, 2, 140000), L.LAP_FD27),
                                       ((64, 262148, 2), L.LAP_FD27), ((2, 524300, 2), L.LAP_FD27)])
def test_stencil_step_and_energies(engine, shape, lap, prec, tol):
    """Two leapfrog steps and the energies on the untuned tile.  FP64: sums of 27 terms of order one, a few
    steps; FP32: the same to the format, energies as sums of FP32 terms."""
    nx, ny, nz = shape
    c = (-6.0, 1.0, 0.0, 0.0, 1.0) if lap == L.LAP_FD7 else (-128.0, 14.0, 3.0, 1.0, 30.0)
    g = engine.Lattice(L.make_config(shape, nfld=1, length=1.0 * nx, laplacian=lap, precision=prec,
                                     model=L.MODEL_PHI4, model_params=(1.0,)))
    dt = 0.05
    f, p = (v[0] for v in random_state((1, nz, ny, nx), seed=11, mean=0.5, amp=0.3))
    g.set_state(f[None], p[None])
    f, p = (v[0] for v in g.get_state())

    def laplacian(v):
        r = neighbours(v, lap)
        return (c[0] * v + sum(w * s for w, s in zip(c[1:], r))) / c[4]

    e = g.energies()
    q = sum(w * (s2 - 2 * f * s1 + k * f * f) for w, s1, s2, k in
            zip(c[1:], neighbours(f, lap), neighbours(f * f, lap), (6, 12, 8)))
    want = {L.E_KE: 0.5 * np.mean(p * p), L.E_GE_LAP: -0.5 * np.mean(f * laplacian(f)),
            L.E_GE_GRAD: 0.25 * np.mean(q) / c[4], L.E_PE: 0.25 * np.mean(f ** 4), L.E_MEAN0: np.mean(f)}
    for i, v in want.items():
        assert abs(e[i] - v) <= tol * abs(v), i
    for s in range(2):
        f = f + dt * p * (0.5 if s == 0 else 1.0)
        p = p + dt * (laplacian(f) - f ** 3)
    f = f + 0.5 * dt * p
    g.symp(2, dt, 2)
    F, P = (v[0] for v in g.get_state())
    assert np.max(np.abs(F - f)) <= tol and np.max(np.abs(P - p)) <= tol
    g.close()
