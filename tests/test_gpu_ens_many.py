"""Energies of an ensemble of more runs than a grid has blocks along y (65535),
against numpy: FP64 sums of 64 sites to rounding, FP32 ones to that of their terms."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(L.FP64, 1e-12), (L.FP32_KAHAN, 1e-5)])
def test_energies_of_many_runs(engine, prec, tol):
    length, sizes = 20.0, [4] * 65540 + [6]
    base = L.make_config(4, nfld=1, length=length, laplacian=L.LAP_SPECTRAL, precision=prec, model=L.MODEL_PHI4,
                         model_params=(1.0,))
    ens = engine.Ensemble(base, sizes)
    ens.init_vacuum(list(range(len(sizes))), 0.8, -0.5, 3.0, amp=100.0, kcut_frac=1.0)
    e = ens.energies()
    assert len(e) == len(sizes)
    for r in (0, 1, 4097, 65534, 65535, 65536, 65539, 65540):
        f, p = ens.state(r)
        f, p, n = f.reshape([sizes[r]] * 3), p.reshape([sizes[r]] * 3), sizes[r]
        k = np.fft.fftfreq(n, 1.0 / n) * 2 * np.pi / length
        k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
        grad = 0.5 * np.sum(k2 * np.abs(np.fft.fftn(f)) ** 2) / float(n) ** 6
        want = {L.E_KE: 0.5 * np.mean(p ** 2), L.E_GE_LAP: grad, L.E_PE: np.mean(f ** 4) / 4, L.E_MEAN0: np.mean(f)}
        for i, v in want.items():
            assert abs(e[r][i] - v) <= tol * abs(v) and abs(v) > 0, (r, i)
