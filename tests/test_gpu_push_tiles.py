"""Large generated networks under push delivery: which of them hold the tiled copy beside their rows,
which cycles are delivered from it (counted on the device), and that nothing else depends on it."""
import numpy as np
import pytest

import bsim_b200 as B
from bsim_b200 import workloads as W

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)


def test_busy_cycles_are_delivered_tiled_and_counted():
    sp = W.cuba(12, 6500, 2000, 6, seed=5)
    out = []
    for bt in (0, -1):
        eng = B.Engine.generated(sp, DT, opts=B.options(build_tiles=bt))
        tiled = []
        for _ in range(60):  # from rest: the first cycles deliver little
            c0 = eng.info().tile_cycles
            eng.run(1)
            tiled.append(eng.info().tile_cycles - c0)
        out.append((eng.fire_count(), eng.state(), eng.info(), tiled))
        eng.close()
    (fa, sa, ia, ta), (fb, sb, ib, tb) = out
    assert ia.n_tiles > 0 and not any(ta[:2]) and 0 < sum(ta) < 60
    assert ib.n_tiles == 0 and not any(tb)
    assert np.array_equal(fa, fb) and fa.sum() > 0 and ia.events_total == ib.events_total
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)


@pytest.mark.parametrize("n_pop,pop,D,synapses,tile_size", [
    (4, 200000, 20, 6e7, 0),     # a tenth of an entry per segment: scanning them costs more than pushing
    (10, 160000, 64, 5.6e7, 256),  # 7e10 segment starts: more than the device's memory
])
def test_sparse_networks_keep_the_rows_alone(n_pop, pop, D, synapses, tile_size):
    sp = W.cuba(n_pop, pop, 2000, D, seed=6)
    sp.p_conn = synapses / (n_pop - 1 + int(0.2 * n_pop + 0.5)) / pop ** 2
    eng = B.Engine.generated(sp, DT, opts=B.options(tile_size=tile_size))
    eng.run(10)
    i = eng.info()
    assert i.n_synapses > 5e7 and i.n_tiles == 0 and i.tile_cycles == 0 and i.events_total > 0
    assert i.device_bytes < 16.5 * i.n_synapses + 400.0 * i.n_neurons + 8.5 * i.n_neurons * D + 1e8
    eng.close()


def test_the_copy_is_not_a_mode_of_its_own():
    """The autotuner keeps a push engine's delivery, its trials push every cycle, and there is no tile to stall."""
    eng = B.Engine.generated(W.cuba(12, 6500, 2000, 6, seed=5), DT)
    assert eng.info().n_tiles > 0
    eng.run(30)
    before = eng.info().tile_cycles
    r = eng.autotune(2)
    i = eng.info()
    assert r.delivery == B.DELIVERY_PUSH and i.delivery == B.DELIVERY_PUSH and i.tile_cycles == before
    assert r.cost_tile[1] == 0.0 and r.cost_push[1] > 0.0
    with pytest.raises(B.BsimError):
        B._check(B.lib().bsim_stall_tile(eng._h, 0))
    eng.run(30)
    assert eng.info().tile_cycles > before
    eng.close()
