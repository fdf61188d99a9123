"""Which networks run many cycles per launch, and the long rows of those that do."""
import numpy as np
import pytest

import bsim_b200 as B
from bsim_b200 import workloads as W
from test_gpu_loop import network, reference, same

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)


@pytest.mark.parametrize("n_pop,pop,p,form", [
    (10, 1000, 0.1, 1), (4, 9000, 0.1, 1),
    (12, 3000, 0.5, 0),  # many synapses
    (3, 3000, 1.0, 0),   # long rows
    (40, 1000, 0.1, 0),  # many neurons
])
def test_networks_with_long_rows_take_one_launch_per_cycle(n_pop, pop, p, form):
    sp = W.cuba(n_pop, pop, 500, 6, seed=3)
    sp.p_conn = p
    sp.w_max *= 0.1 / p
    out = []
    for delivery in (B.DELIVERY_PUSH, B.DELIVERY_TILE, B.DELIVERY_AUTO):
        eng = B.Engine.generated(sp, DT, opts=B.options(delivery=delivery))
        eng.run(40)
        i = eng.info()
        assert i.many_cycles == form
        if delivery != B.DELIVERY_PUSH:  # (a large push engine may hold tiles for its busy cycles)
            assert i.tile_cycles == (40 if delivery == B.DELIVERY_TILE and form == 0 else 0)
        out.append((eng.fire_count(), eng.state()["v"], i.events_total))
        eng.close()
    for f, v, ev in out[1:]:
        assert np.array_equal(f, out[0][0]) and np.array_equal(v, out[0][1]) and ev == out[0][2]
    assert out[0][0].sum() > 0
    if n_pop * pop < 37888:
        eng = B.Engine.generated(sp, DT, opts=B.options(delivery=B.DELIVERY_PULL))
        eng.run(40)
        assert eng.info().many_cycles == 2 and np.array_equal(eng.fire_count(), out[0][0])
        eng.close()


@pytest.mark.parametrize("burst", [False, True])
@pytest.mark.parametrize("n,D,degree", [(150, 64, 1037), (700, 1, 515), (700, 2, 511), (2000, 5, 257), (1, 3, 2049)])
def test_long_rows_equal_the_oracle(n, D, degree, burst):
    """Rows of more and fewer pairs than one pass of a warp, from odd and even positions, whole and cut
    among warps, with one delay, a few, and more delays than entries of a segment."""
    net = network(n, D, degree, seed=n + degree, burst=burst)
    net[3][:] *= np.float32(20.0 / degree)
    steps = 50
    eng = B.Engine.from_arrays(*net, DT)
    eng.record(steps, n * steps)
    eng.run(steps)
    assert eng.info().many_cycles == 1
    ref = reference(net, steps, eng)
    assert ref["fire_count"].sum() > 0
    same(eng, ref, steps)
    eng.close()
