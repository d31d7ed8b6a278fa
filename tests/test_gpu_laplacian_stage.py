"""Laplacian read-out of a fresh one-field stencil lattice: its FP64 copy and its
result lie side by side in the stage, which uploads had made for one array only."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import L, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(L.FP64, 1e-13), (L.FP32_KAHAN, 1e-6)])
@pytest.mark.parametrize("shape", [(15, 9, 21), (96, 80, 64), (160, 160, 160)])
def test_fresh_lattice(engine, shape, prec, tol):
    """FP64 sums of seven terms; an FP32 field is its leading part, phi to 2^-25."""
    nx, ny, nz = shape
    g = engine.Lattice(L.make_config(shape, nfld=1, length=1.0 * nx, laplacian=L.LAP_FD7, precision=prec,
                                     model=L.MODEL_PHI4, model_params=(1.0,)))
    g.set_state(*random_state((1, nz, ny, nx), seed=3, mean=0.5, amp=1.0))
    got = g.laplacian()
    f = g.get_state()[0][0]
    ref = sum(np.roll(f, s, d) for s in (1, -1) for d in (0, 1, 2)) - 6 * f
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref))
    g.close()
