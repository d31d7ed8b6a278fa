"""Two-field lattices whose second field starts off a 16-byte boundary."""
from __future__ import annotations

import pytest

from conftest import rel_err
from helpers import L, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [L.FP64, L.FP32_KAHAN])
@pytest.mark.parametrize("lap", [L.LAP_SPECTRAL, L.LAP_FD7])
@pytest.mark.parametrize("shape", [(9, 11, 13), (10, 11, 13), (12, 11, 13)])
def test_two_fields_whose_arrays_start_unaligned(engine, orc, shape, lap, prec):
    """With an odd number of sites (FP32: not a multiple of four) the second field's array starts
    off a 16-byte boundary: the pointwise passes then move one site at a time."""
    nx, ny, nz = shape
    c = L.make_config(shape, nfld=2, length=0.5 * nx, laplacian=lap, background=L.BG_CONFORMAL, precision=prec,
                      model=L.MODEL_PHI4_G2, model_params=(1.0, 2.0))
    c64 = L.make_config(shape, nfld=2, length=0.5 * nx, laplacian=lap, background=L.BG_CONFORMAL, precision=L.FP64,
                        model=L.MODEL_PHI4_G2, model_params=(1.0, 2.0))
    g, o = engine.Lattice(c), orc.Oracle(c64)
    f, p = random_state((2, nz, ny, nx), seed=2, mean=0.7, amp=0.1)
    for h in (g, o):
        h.set_state(f, p)
        h.set_scale_factor(1.0, -0.3)
        h.symp(4, 0.02, 4)
    tol = 1e-12 if prec == L.FP64 else 1e-5
    (fg, pg), (fo, po) = g.get_state(), o.get_state()
    assert rel_err(fg, fo) <= tol and rel_err(pg, po) <= 10 * tol
    assert abs(g.scale_factor()[1] - o.scale_factor()[1]) <= tol * abs(o.scale_factor()[1])
