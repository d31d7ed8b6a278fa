"""Long thin and wide boxes: shapes whose longest side is far beyond the others.

Spectra of sides beyond 4096 points, which hold |n|^2 past the last shell (2047),
against numpy.  Counts and weights hold no data: they agree to rounding.  A bin's
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
