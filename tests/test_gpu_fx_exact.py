"""FP64 spectral runs on the fixed-point passes and on cuFFT, both against the same
steps in the platform's long double (quad on Arm): the passes are no further off.

Two Yoshida-4 steps from the engine's own vacuum; the line derivatives are dense
sums.  Fields are dominated by the rounding of their own storage, equal on both
sides; momenta by the transforms.  5% covers the spread of the figures over some
30000 sites (0.4%) several times.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import L

pytestmark = pytest.mark.gpu
LD = np.longdouble


def second_derivative(n):
    """Matrix of a line's derivative for dk = 1."""
    f = np.minimum(np.arange(n), n - np.arange(n)).astype(LD)
    j = np.arange(n)
    # 8 atan(1): 2 pi in long double
    ang = 8 * np.arctan(LD(1)) * (np.outer(j, j) % n).astype(LD) / n
    c = -(np.cos(ang) * f * f).sum(1) / n
    return c[(j[:, None] - j[None, :]) % n]


@pytest.mark.skipif(np.finfo(LD).eps > 1e-18, reason="no long double beyond FP64")
@pytest.mark.parametrize("shape,nf", [((32, 32, 32), 2), ((50, 36, 32), 1), ((33, 40, 27), 2)])
def test_no_further_off_than_cufft(engine, shape, nf):
    nx, ny, nz = shape
    length = 10 * np.pi if nf == 2 else 20.0
    dt = length / nx / 20
    state, runs = None, {}
    for impl in (L.SPEC_IMPL_AUTO, L.SPEC_IMPL_CUFFT):
        g = engine.Lattice(L.make_config(shape, nfld=nf, length=length, laplacian=L.LAP_SPECTRAL, precision=L.FP64,
                                         model=L.MODEL_PHI4_G2 if nf == 2 else L.MODEL_PHI4,
                                         model_params=(1.0, 2.0) if nf == 2 else (1.0,), spectral_impl=impl))
        if state is None:
            g.init_vacuum(5, [0.8, 0.0][:nf], [-0.5, 0.0][:nf], [3.0, 2.0][:nf], amp=1e-8, kcut_frac=0.5)
            state = g.get_state()
        g.set_state(*state)
        assert g.tuning()[5] == (L.SPEC_IMPL_CUFFT if impl == L.SPEC_IMPL_CUFFT else L.SPEC_IMPL_SEPARABLE)
        g.symp(4, dt, 2)
        runs[impl] = g.get_state()
        g.close()
    dk = [LD(2 * np.pi / (n * (length / nx))) for n in (nz, ny, nx)]  # as the engine has them
    mats = [second_derivative(n) * k * k for n, k in zip((nz, ny, nx), dk)]
    f, p = (v.astype(LD) for v in state)

    def force(f):
        out = np.zeros_like(f)
        for i in range(nf):
            for ax, m in enumerate(mats):
                out[i] += np.moveaxis(np.tensordot(m, f[i], axes=(1, ax)), 0, ax)
        return out - (np.stack([f[0] ** 3 + 2 * f[0] * f[1] ** 2, 2 * f[0] ** 2 * f[1]]) if nf == 2 else f ** 3)

    w1 = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
    w = [w1, 1.0 - 2.0 * w1, w1]
    f = f + p * (LD(w[0]) * LD(dt) / 2)
    for s in range(2):
        for i in range(3):
            p = p + LD(w[i]) * LD(dt) * force(f)
            nxt = w[i + 1] if i < 2 else (w[0] if s == 0 else 0.0)
            f = f + p * ((LD(w[i]) + LD(nxt)) * LD(dt) / 2)
    for i in range(nf):
        for k, ref in ((0, f[i]), (1, p[i])):
            off = [float(np.sqrt(np.sum((runs[m][k][i] - ref) ** 2))) for m in (L.SPEC_IMPL_AUTO, L.SPEC_IMPL_CUFFT)]
            assert off[0] <= 1.05 * off[1], (i, k, off)
            assert off[1] <= 1e-14 * float(np.sqrt(np.sum(ref ** 2)))
