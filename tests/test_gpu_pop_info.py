"""Population degrees of engines that hold the tiled copy alone, with populations that share
tiles, against the host generator's synapse lists."""
import numpy as np
import pytest

import bsim_b200 as B
from bsim_b200 import workloads as W

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)


def degrees(specs):
    want_in, want_out = [], []
    for sp in specs:
        g = B.gen_host(sp)
        want_in += list(np.bincount(g["pop"][g["dst"]], minlength=sp.n_pop) / sp.pop_size)
        want_out += list(np.bincount(g["pop"][g["src"]], minlength=sp.n_pop) / sp.pop_size)
    return want_in, want_out


@pytest.mark.parametrize("specs,tile_size", [
    ([W.cuba(100, 500, 500, 6, seed=3)], 0),  # two populations to a tile by the engine's own tile size
    ([W.cuba(9, 130, 500, 6, seed=4), W.cuba(5, 700, 100, 30, seed=5), W.cuba(40, 33, 100, 3, seed=6)], 400),
    ([W.cuba(6, 90, 100, 6, seed=7)], 12288),  # one tile for the network
    ([W.cuba(4, 300, 100, 6, seed=8)], 256),  # populations cut into tiles of their own
])
def test_degrees_of_populations_that_share_tiles(specs, tile_size):
    # a fixed launch shape: one launch per cycle at every size, so no push rows are held
    eng = B.Engine.generated(specs, DT, opts=B.options(delivery=B.DELIVERY_TILE, tile_size=tile_size,
                                                       block_threads=512))
    size, indeg, outdeg = eng.pop_info()
    want_in, want_out = degrees(specs)
    assert list(size) == [sp.pop_size for sp in specs for _ in range(sp.n_pop)]
    assert np.allclose(indeg, want_in, rtol=1e-6) and np.allclose(outdeg, want_out, rtol=1e-6)
    eng.close()
