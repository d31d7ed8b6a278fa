"""FP32 gradient energies keep what the compensated sum can hold.

On a 4^3 lattice every twiddle is 1 or i, so the FP32 transform of whole numbers
is exact, and with dk = 1 so is every term w k^2 |F|^2.  Mirrored rows hold modes
of very different size (their terms' ratio is beyond 2^24): the compensated sum
is exact, while any sum of two rows in plain FP32 loses the smaller one, 2^-26 to
2^-30 of the energy.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

from helpers import L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big,small", [(8192, 1), (8192, 3), (32768, 1)])
def test_rows_of_different_size(engine, big, small):
    n = 4
    g = engine.Lattice(L.make_config(n, nfld=1, length=2 * math.pi, laplacian=L.LAP_SPECTRAL, precision=L.FP32_KAHAN,
                                     model=L.MODEL_PHI4, model_params=(1.0,)))
    z, y, x = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    cos = lambda m: np.array([1.0, 0.0, -1.0, 0.0])[m % 4]  # noqa: E731
    f = big * cos(x + y) + small * cos(x - y) + small * cos(x + y + z) + small * cos(x - y + z)
    g.set_state(f[None], np.zeros((1, n, n, n)))
    assert np.array_equal(g.get_state()[0][0], f)
    # mean of the squared gradient: amplitude^2 / 2 times |n|^2
    want = 0.5 * (2 * big ** 2 + 2 * small ** 2 + 2 * 3 * small ** 2) / 2
    got = g.energies()[L.E_GE_LAP]
    assert abs(got - want) <= 1e-13 * want
    g.close()
