"""Read-outs of both fields of lattices with an odd number of sites, whose second
arrays start off a 16-byte boundary: power and cross spectra and the Laplacian.

Spectra are FP64 transforms of the fields as the engine holds them (1e-11 of a
bin's absolute sum, as everywhere); the FP32 Laplacian is an FP32 transform pair,
1e-5 of its largest value on noise."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import L, random_state
from test_gpu_bins import two_bin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
@pytest.mark.parametrize("lap", [L.LAP_SPECTRAL, L.LAP_FD7])
@pytest.mark.parametrize("shape", [(15, 9, 21), (9, 3, 5), (65, 9, 11), (18, 9, 11)])
def test_second_field(engine, shape, lap, prec):
    nx, ny, nz = shape
    length = 3.0
    g = engine.Lattice(L.make_config(shape, nfld=2, length=length, laplacian=lap, precision=prec,
                                     model=L.MODEL_PHI4_G2, model_params=(1.0, 2.0)))
    g.set_state(*random_state((2, nz, ny, nx), seed=7, mean=0.3, amp=1.0))
    f, p = g.get_state()
    nb = 12
    F = {(w, i): np.fft.rfftn(v[i]).ravel() for w, v in ((L.SPEC_FLD, f), (L.SPEC_FLDP, p)) for i in (0, 1)}
    W = two_bin(shape, np.ones(F[L.SPEC_FLD, 0].size), nb)
    ok = W != 0
    for k, v in F.items():
        S, _ = g.spectrum(*k, L.SPEC_WEIGHTED, nb)
        assert np.allclose(S[ok] * W[ok], two_bin(shape, np.abs(v) ** 2, nb)[ok], rtol=1e-11, atol=0), k
    for a in F:
        for b in F:
            x = F[a] * F[b].conj()
            size = two_bin(shape, np.abs(x), nb)
            for got, v in zip(g.crossspec_3d(*a, *b, nb), (x.real, x.imag)):
                assert np.all(np.abs(got[ok] * W[ok] - two_bin(shape, v, nb)[ok]) <= 1e-11 * size[ok]), (a, b)
    dx = length / nx
    for i in (0, 1):
        if lap == L.LAP_FD7:
            ref = (sum(np.roll(f[i], s, d) for s in (1, -1) for d in (0, 1, 2)) - 6 * f[i]) / dx ** 2
        else:
            k = [np.fft.fftfreq(n, 1.0 / n) * 2 * np.pi / (n * dx) for n in (nz, ny, nx)]
            k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
            ref = np.fft.ifftn(-k2 * np.fft.fftn(f[i])).real
        tol = 1e-12 if prec == L.FP64 else 1e-5
        assert np.max(np.abs(g.laplacian(i) - ref)) <= tol * np.max(np.abs(ref)), i
    g.close()
