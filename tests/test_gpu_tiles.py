"""Tiled delivery at the places where its listing and its shared-memory ring can go
wrong, against the oracle (EXACT accumulation: spikes, state and events equal)."""
import numpy as np
import pytest

import bsim_b200 as B
from oracle import oracle

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)
LIF = [-0.065, -0.065, -0.065, 0.25e-9, 20e-3, 0.3e-3, 5e-3, 10e-3, -0.050, 0.0]


def network(n, seed):
    """Sources in runs of 1, 2, 31, 32, 33 and 70 consecutive ids with gaps between them, each
    with 0, 1, 2 or many synapses per delay (so a listing holds empty, single-pair and long
    segments), some weights +0.0 and -0.0, most neurons firing every few cycles."""
    rng = np.random.default_rng(seed)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:, 0] = rng.uniform(-0.065, -0.051, n)
    params[:, 9] = rng.uniform(1e-9, 40e-9, n)
    sources, at = [], 3
    for k in [1, 2, 31, 32, 33, 70]:
        sources += range(at, at + k)
        at += k + 5
    assert at < n
    src, dst, w, d = [], [], [], []
    for s in sources:
        for delay in (1, 2, 5, 9):
            k = int(rng.choice([0, 1, 2, 3, 40, 150]))
            src += [s] * k
            dst += rng.integers(0, n, k).tolist()
            w += rng.uniform(-2e-10, 1.5e-10, k).tolist()
            d += [delay] * k
    w = np.asarray(w, np.float32)
    w[::17], w[5::17] = 0.0, -0.0
    return params, np.asarray(src, np.int32), np.asarray(dst, np.int32), w, np.asarray(d, np.int32)


@pytest.mark.parametrize("tile_size", [256, 1000, 12288])
@pytest.mark.parametrize("block", [0, 32, 480])
def test_tiled_listing_edges(tile_size, block):
    n, steps = 2300, 150
    params, src, dst, w, d = network(n, seed=tile_size + block)
    eng = B.Engine.from_arrays(params, src, dst, w, d, DT,
                               opts=B.options(delivery=B.DELIVERY_TILE, tile_size=tile_size, block_threads=block,
                                              graph_steps=0))  # cycle by cycle: the tiled kernel at this size
    eng.record(steps, n * steps)
    eng.run(steps)
    ref = oracle.run(params, src, dst, w, d, DT, steps, record_steps=steps, acc_mode=oracle.ACC_FIXED,
                     qexp=int(eng.qexp()[0]), raster_cap=n * steps)
    assert ref["events_per_step"].max() > 2000
    for t, (a, b) in enumerate(zip(eng.raster(), ref["raster"])):
        assert np.array_equal(a, b), t
    assert np.array_equal(eng.state()["v"], ref["final_state"][:, 0])
    assert eng.info().events_total == ref["events_per_step"].sum()
    eng.close()


def test_largest_tile_fits():
    """A tile of 12,288 targets (the largest accepted) leaves the warps' rings their shared memory."""
    n, steps = 12288, 40
    rng = np.random.default_rng(4)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:, 9] = rng.uniform(5e-9, 40e-9, n)
    src, dst = rng.integers(0, n, 20 * n).astype(np.int32), rng.integers(0, n, 20 * n).astype(np.int32)
    w, d = rng.uniform(-2e-10, 2e-10, 20 * n).astype(np.float32), rng.integers(1, 4, 20 * n).astype(np.int32)
    eng = B.Engine.from_arrays(params, src, dst, w, d, DT, opts=B.options(delivery=B.DELIVERY_TILE, tile_size=12288, graph_steps=0))
    eng.run(steps)
    ref = oracle.run(params, src, dst, w, d, DT, steps, acc_mode=oracle.ACC_FIXED, qexp=int(eng.qexp()[0]))
    assert np.array_equal(eng.fire_count(), ref["fire_count"])
    assert np.array_equal(eng.state()["v"], ref["final_state"][:, 0])
    assert eng.info().events_total == ref["events_per_step"].sum() > 0
    eng.close()


@pytest.mark.parametrize("length", [1, 3, 255, 256, 257, 300])
def test_segment_lengths_and_small_populations_in_one_tile(length):
    """Segments around the bank ordering's limit, populations of 7 to 90 neurons sharing tiles, a
    population without sources, two networks in one engine (tiles do not straddle them)."""
    sizes, nets = [7, 30, 90, 41, 12, 60, 700], [0, 0, 0, 0, 1, 1, 1]
    n, steps = sum(sizes), 120
    rng = np.random.default_rng(length)
    pop = np.repeat(np.arange(7), sizes).astype(np.int32)
    inst = np.repeat(nets, sizes).astype(np.int32)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:, 9] = rng.uniform(2e-9, 30e-9, n)
    src, dst, w, d = [], [], [], []
    for a, b in ((0, 1), (0, 2), (1, 2), (2, 3), (4, 5), (5, 6), (6, 6)):
        s, t = np.nonzero(pop == a)[0], np.nonzero(pop == b)[0]
        for x in s:
            k = min(length, len(t))
            src += [x] * k
            dst += rng.choice(t, k, replace=False).tolist()
            d += [1 + x % 3] * k
    w = rng.uniform(-2e-10, 2e-10, len(src)).astype(np.float32)
    src, dst, d = (np.asarray(v, np.int32) for v in (src, dst, d))
    eng = B.Engine.from_arrays(params, src, dst, w, d, DT, pop=pop, instance=inst,
                               opts=B.options(delivery=B.DELIVERY_TILE, tile_size=600, graph_steps=0))
    eng.run(steps)
    q = eng.qexp()
    ref = oracle.run(params, src, dst, w, d, DT, steps, acc_mode=oracle.ACC_FIXED, qexp=q[inst], instance=inst)
    assert np.array_equal(eng.fire_count(), ref["fire_count"]) and ref["fire_count"].sum() > 0
    assert np.array_equal(eng.state()["v"], ref["final_state"][:, 0])
    assert eng.info().events_total == ref["events_per_step"].sum()
    # the many-cycle launch gives the same
    loop = B.Engine.from_arrays(params, src, dst, w, d, DT, pop=pop, instance=inst,
                                opts=B.options(delivery=B.DELIVERY_TILE))
    loop.run(steps)
    assert np.array_equal(loop.fire_count(), ref["fire_count"])
    assert loop.info().events_total == eng.info().events_total


def test_busy_cycles_of_a_large_pushed_network():
    """A generated network large enough to hold the tiled copy beside its push rows: quiet cycles are
    pushed, busy ones tiled, with the spikes, state and events of the rows alone (build_tiles = -1)."""
    from bsim_b200 import workloads as W
    sp = W.cuba(12, 6500, 2000, 6, seed=5)
    out = []
    for bt in (0, -1):
        eng = B.Engine.generated(sp, DT, opts=B.options(build_tiles=bt))
        per = []
        for n in [1] * 8 + [10] * 12:  # the first cycles' deliveries grow from nothing
            e0 = eng.info().events_total
            eng.run(n)
            per.append((eng.info().events_total - e0) / n)
        out.append((eng.fire_count(), eng.state(), per, eng.info().device_bytes))
        eng.close()
    (fa, sa, pa, ba), (fb, sb, pb, bb) = out
    assert ba > 1.5 * bb  # both copies were held
    assert min(pa) < 3e6 and max(pa) > 9e6  # both modes ran
    assert pa == pb and np.array_equal(fa, fb)
    assert all(np.array_equal(sa[k], sb[k]) for k in sa)
