"""FP64 stencil steps with rolling plane sums: the split of the planes over blocks
does not enter the arithmetic, so any tile gives the same bits, down to chunks
of one and two planes and blocks wider than the lattice."""
from __future__ import annotations

import json

import numpy as np
import pytest

from helpers import L

pytestmark = pytest.mark.gpu


def _state(engine, shape, gw, nf, tile, tmp):
    cfg = L.make_config(shape, nfld=nf, length=8.0, laplacian=27, background=0, precision=0,
                        split_order=1 if gw else 0, model=2 if gw and nf == 1 else (1 if nf == 2 else 0),
                        model_params=(0.01,) if gw and nf == 1 else (1.0, 2.0), gw=gw, gw_coupling=2.0 if gw else 0.0)
    g = L.Lattice(cfg)
    if tile:
        path = str(tmp / ("t%d_%d.json" % tile))
        probe = L.Lattice(cfg)
        probe.autotune(path)
        rec = json.loads(open(path).read().splitlines()[-1])
        probe.close()
        rec["ty"], rec["zc"] = tile
        with open(path, "w") as f:
            f.write('{"key": "%s", "ty": %d, "zc": %d, "pw_block": %d, "pw_bps": %d, "sep": 0}\n'
                    % (rec["key"], tile[0], tile[1], rec["pw_block"], rec["pw_bps"]))
        g.autotune(path)
        assert tuple(g.tuning()[1:3]) == tile
    rng = np.random.default_rng(3)
    if gw:
        g.set_gw_state(*rng.standard_normal((2, 6) + shape[::-1]))
    fld = rng.standard_normal((nf,) + shape[::-1])
    g.set_state(fld, 0.1 * rng.standard_normal(fld.shape))
    g.symp(2, 1e-3, 3)
    out = [np.array(v) for v in g.get_state()]
    if gw:
        out += [np.array(v) for v in g.gw_state()]
    g.close()
    return out


@pytest.mark.parametrize("gw,nf", [(0, 1), (1, 1), (0, 2), (1, 2)])
@pytest.mark.parametrize("shape", [(34, 9, 7), (16, 6, 3)])
def test_tiles_give_the_same_bits(engine, shape, gw, nf, tmp_path):
    ref = _state(engine, shape, gw, nf, None, tmp_path)
    for tile in ((2, 2), (8, 3), (4, shape[2])):
        for a, b in zip(ref, _state(engine, shape, gw, nf, tile, tmp_path)):
            assert np.array_equal(a, b), tile
