"""Gradients of the closure with fewer tiles than blocks, with exactly one round
of them, and with rounds that end unevenly (the tiles of a block alternate
between two slots); on 64-site rows also the tensor-memory convolutions with
runs of planes that cross columns and that are longer than a column."""
from __future__ import annotations

import numpy as np
import pytest

import net_oracle as NO
from conftest import rel_err
from test_gpu_closure import _dataset, _net

pytestmark = pytest.mark.gpu


# (sites, samples): 16 x 8 sites of one plane are a tile
@pytest.mark.parametrize("shape,idx", [((16, 8, 1), [0]), ((48, 24, 17), [1]), ((32, 8, 1), [1]), ((96, 24, 2), [0, 1]), ((64, 16, 19), [1, 0, 1]),
                                       ((64, 64, 3), [0, 1, 1, 0, 1, 0, 0, 1, 1, 0, 1])])
def test_gradients_over_uneven_rounds(engine, shape, idx):
    host, buf = _dataset(engine, shape, 2, 21)
    net, p, norm = _net(engine, 23)
    loss, g = net.grad(buf, 6 * int(np.prod(shape)), idx, shape)
    lref, gref = NO.loss_and_grad(p, host[idx], norm, emulate=True)
    # as for the other gradients: FP32 sums of BF16 products, so only flips of a
    # BF16 rounding (2^-9 of single activations) tell the two apart
    assert abs(loss - lref) <= 1e-3 * lref
    off = 0
    for name, shp in NO.SHAPES:
        n = int(np.prod(shp))
        live = NO.mask()[off:off + n] > 0
        assert rel_err(g[off:off + n][live], gref[off:off + n][live]) <= 2e-2, name
        assert np.all(g[off:off + n][~live] == 0), name
        off += n
