"""Small networks run many cycles per launch: the same spikes, state, counts, events,
recording, trace and statistics as one launch per cycle (graph_steps = 0) and as the
oracle, for any split of a run into calls and when the two ways alternate."""
import numpy as np
import pytest

import bsim_b200 as B
from oracle import oracle

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)
LIF = [-0.065, -0.065, -0.065, 0.25e-9, 20e-3, 0.5e-3, 5e-3, 10e-3, -0.050, 0.0]


def network(n, D, degree, seed, burst=False):
    rng = np.random.default_rng(seed)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:, 0] = -0.0505 if burst else rng.uniform(-0.065, -0.051, n)
    params[:, 9] = 8e-9 if burst else rng.uniform(0.3e-9, 12e-9, n)
    s = n * degree
    src, dst = rng.integers(0, n, s).astype(np.int32), rng.integers(0, n, s).astype(np.int32)
    w = rng.uniform(-3e-10, 3e-10, s).astype(np.float32)
    d = rng.integers(1, D + 1, s).astype(np.int32)
    return params, src, dst, w, d


def reference(net, steps, eng):
    return oracle.run(*net, DT, steps, record_steps=steps, acc_mode=oracle.ACC_FIXED, qexp=int(eng.qexp()[0]),
                      raster_cap=net[0].shape[0] * steps)


def same(eng, ref, steps):
    raster = eng.raster()
    assert len(raster) == steps
    for t in range(steps):
        assert np.array_equal(raster[t], ref["raster"][t]), t
    assert np.array_equal(eng.state()["v"], ref["final_state"][:, 0])
    assert np.array_equal(eng.fire_count(), ref["fire_count"])
    assert eng.info().events_total == ref["events_per_step"].sum()


@pytest.mark.parametrize("delivery", [B.DELIVERY_PUSH, B.DELIVERY_PULL])
@pytest.mark.parametrize("n,D,degree", [(1, 1, 3), (7, 2, 4), (33, 64, 30), (1007, 1, 9), (1500, 6, 40), (9473, 3, 5)])
def test_any_split_of_a_run_equals_the_oracle(n, D, degree, delivery):
    net = network(n, D, degree, seed=n + D)
    steps = 120
    eng = B.Engine.from_arrays(*net, DT, opts=B.options(delivery=delivery))
    eng.record(steps, n * steps)
    for k in (1, 2, 3, 1, 1, 40, 7, 65):
        eng.run(k)
    ref = reference(net, steps, eng)
    assert ref["fire_count"].sum() > 0
    same(eng, ref, steps)
    eng.close()


@pytest.mark.parametrize("n", [4736, 4737, 300 * 32 + 5])
def test_populations_that_fire_together(n):
    """Every neuron fires in the same cycles: full spike lists in every block, long rows in few cycles."""
    net = network(n, 2, 30, seed=n, burst=True)
    eng = B.Engine.from_arrays(*net, DT)
    eng.record(60, n * 60)
    eng.run(60)
    ref = reference(net, 60, eng)
    assert ref["spikes_per_step"].max() >= 0.9 * n
    same(eng, ref, 60)
    eng.close()


def test_alternating_with_one_launch_per_cycle():
    """The autotuner's trials launch cycle by cycle: spikes in flight, the recording and the event
    count pass from one way to the other and back."""
    net = network(2000, 9, 25, seed=3)
    eng = B.Engine.from_arrays(*net, DT)
    eng.record(400, 2000 * 400)
    eng.run(25)
    eng.autotune(2)
    eng.run(31)
    eng.autotune(1)
    eng.run(2)
    steps = int(eng.info().steps_done)
    same(eng, reference(net, steps, eng), steps)
    eng.close()


@pytest.mark.parametrize("ordered", [False, True])
def test_trace_and_statistics_equal_one_launch_per_cycle(ordered):
    n, steps = 1300, 70
    params, src, dst, w, d = network(n, 5, 20, seed=8)
    pop = (np.arange(n) // 100).astype(np.int32)
    out = []
    for gs in (0, 64):
        o = B.options(graph_steps=gs, accumulate=B.ACC_ORDERED if ordered else B.ACC_EXACT)
        eng = B.Engine.from_arrays(params, src, dst, w, d, DT, pop=pop, opts=o)
        eng.enable_pop_stats(80)
        eng.run(11)
        eng.trace(40, 13, 900)
        eng.run(steps - 11)
        out.append((eng.read_trace(), eng.pop_counts(steps), eng.state(), eng.info().events_total))
        eng.close()
    (ta, ca, sa, ea), (tb, cb, sb, eb) = out
    assert all(np.array_equal(ta[k], tb[k]) for k in ta) and ta["v"].shape == (40, 900)
    assert np.array_equal(ca, cb) and ca.sum() > 0 and ea == eb
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)


@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("n,D,degree", [(33, 3, 3000), (9473, 2, 700), (1500, 40, 40), (150, 1, 5)])
def test_rows_held_in_part_or_not_at_all(n, D, degree, ordered):
    """Pull: rows that stay in shared memory, that do in part, and that are too long; launches of one,
    two, an even and an odd number of cycles."""
    net = network(n, D, degree, seed=n)
    net[3][:] *= np.float32(20.0 / degree)
    out = []
    for gs in (0, 64):
        o = B.options(graph_steps=gs, delivery=B.DELIVERY_PULL,
                      accumulate=B.ACC_ORDERED if ordered else B.ACC_EXACT)
        eng = B.Engine.from_arrays(*net, DT, opts=o)
        eng.record(60, n * 60)
        for k in (1, 2, 3, 4, 1, 30, 19):
            eng.run(k)
        out.append((eng.raster(), eng.state(), eng.fire_count(), eng.info().events_total))
        eng.close()
    (ra, sa, fa, ea), (rb, sb, fb, eb) = out
    assert fa.sum() > 0 and ea == eb and np.array_equal(fa, fb)
    assert all(np.array_equal(x, y) for x, y in zip(ra, rb))
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)


@pytest.mark.parametrize("D", [1, 6, 40])
def test_auto_schedule_counts_its_choices(D):
    """Small AUTO engines under the exact schedule: the spikes, events and statistics of one launch per
    cycle, with a choice that changes along the run."""
    net = network(1500, D, 30, seed=D, burst=True)
    out = []
    for gs in (0, 64):
        eng = B.Engine.from_arrays(*net, DT, opts=B.options(graph_steps=gs, delivery=B.DELIVERY_AUTO))
        eng.set_predictor(None, 0.25, (10.0, 6.5), (10000.0, 3.0))
        for k in (1, 2, 40, 7, 50):
            eng.run(k)
        out.append((eng.fire_count(), eng.state(), eng.info().events_total, eng.predictor_stats()))
        eng.close()
    (fa, sa, ea, pa), (fb, sb, eb, pb) = out
    assert fa.sum() > 0 and ea == eb and np.array_equal(fa, fb)
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)
    assert pa.cycles == pb.cycles == 100 and pa.tile_cycles == pb.tile_cycles and 0 < pa.tile_cycles < 100
