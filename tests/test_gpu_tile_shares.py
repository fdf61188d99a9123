"""Tiled delivery's shares over cycles that are unlike one another: 1-step delays with populations that
fire together, cycles pushed between tiled ones, many tiles with few blocks and few tiles with many."""
import numpy as np
import pytest

import bsim_b200 as B
from test_gpu_loop import network, reference, same

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)


@pytest.mark.parametrize("delivery", [B.DELIVERY_TILE, B.DELIVERY_AUTO])
@pytest.mark.parametrize("n,D,degree,tile_size,grid", [(3000, 1, 40, 256, 0), (3000, 1, 40, 256, 3), (700, 1, 60, 12288, 0),
                                                       (2000, 2, 30, 300, 0)])
def test_bursts_equal_the_oracle(n, D, degree, tile_size, grid, delivery):
    net = network(n, D, degree, seed=n + grid, burst=True)
    steps = 90
    eng = B.Engine.from_arrays(*net, DT, opts=B.options(delivery=delivery, tile_size=tile_size, block_threads=512,
                                                        grid_blocks=grid))
    if delivery == B.DELIVERY_AUTO:  # bursts tiled, the cycles between them pushed
        eng.set_predictor(None, 0.25, (0.0, 1.0), (0.3 * n * degree, 0.1))
    eng.record(steps, n * steps)
    for k in (1, 2, 37, 50):
        eng.run(k)
    i = eng.info()
    assert i.many_cycles == 0
    assert i.tile_cycles == steps if delivery == B.DELIVERY_TILE else 0 < i.tile_cycles < steps
    ref = reference(net, steps, eng)
    assert ref["spikes_per_step"].max() >= 0.5 * n
    same(eng, ref, steps)
    eng.close()
