"""The tiled copy at the limits of what it can hold, against the oracle."""
import numpy as np
import pytest

import bsim_b200 as B
from oracle import oracle

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)
LIF = [-0.065, -0.065, -0.065, 0.25e-9, 20e-3, 0.3e-3, 5e-3, 10e-3, -0.050, 0.0]


def engine(net, pop=None, **opt):
    return B.Engine.from_arrays(*net, DT, pop=pop, opts=B.options(delivery=B.DELIVERY_TILE, block_threads=512, **opt))


def same_as_oracle(net, steps, eng):
    n = net[0].shape[0]
    eng.record(steps, n * steps)
    eng.run(steps)
    ref = oracle.run(*net, DT, steps, record_steps=steps, acc_mode=oracle.ACC_FIXED, qexp=int(eng.qexp()[0]),
                     raster_cap=n * steps)
    assert eng.info().tile_cycles == steps and ref["events_per_step"].sum() > 0
    for t, (a, b) in enumerate(zip(eng.raster(), ref["raster"])):
        assert np.array_equal(a, b), t
    assert np.array_equal(eng.state()["v"], ref["final_state"][:, 0])
    assert eng.info().events_total == ref["events_per_step"].sum()
    eng.close()


@pytest.mark.parametrize("lengths", [[1, 2, 3], [4, 31, 40]])
def test_weights_that_vanish_in_fixed_point(lengths):
    """A strong synapse of a silent neuron sets a coarse fixed-point scale, at which other weights
    underflow: they add nothing, but are delivered and counted."""
    n, steps = 200, 60
    rng = np.random.default_rng(5)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:60, 9] = rng.uniform(5e-9, 20e-9, 60)  # these fire; the others never do
    src, dst, w, d = [199], [198], [1e25], [1]
    for s in range(60):
        k = lengths[s % len(lengths)]
        src += [s] * k
        dst += rng.choice(150, k, replace=False).tolist()
        w += rng.choice([-1e-40, 1e-40, -1e-38, -0.0, 0.0, -2e-10, 1e-10], k).tolist()
        d += [1 + s % 4] * k
    net = (params, np.asarray(src, np.int32), np.asarray(dst, np.int32), np.asarray(w, np.float32), np.asarray(d, np.int32))
    same_as_oracle(net, steps, engine(net))


@pytest.mark.parametrize("per_pop,D", [((40000, 40000), 3), ((65534, 0), 1), ((33000, 65532), 2)])
def test_a_source_with_many_synapses(per_pop, D):
    """The limit of 65,535 synapses of one source into a range of targets counts populations apart, also
    where two of them share a tile."""
    n, steps = 60, 40
    rng = np.random.default_rng(D)
    pop = (np.arange(n) >= 40).astype(np.int32)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[0, 9] = 12e-9
    src, dst, d = [], [], []
    for p, k in enumerate(per_pop):
        src += [0] * k
        dst += rng.choice(np.nonzero(pop == p)[0], k).tolist()
        d += (1 + np.arange(k) % D).tolist()
    w = rng.uniform(-1e-15, 3e-15, len(src))
    net = (params, np.asarray(src, np.int32), np.asarray(dst, np.int32), np.asarray(w, np.float32), np.asarray(d, np.int32))
    same_as_oracle(net, steps, engine(net, pop=pop))


@pytest.mark.parametrize("count,D", [(65536, 1), (65535, 1), (65534, 3)])
def test_a_source_over_the_limit_is_refused(count, D):
    n = 60
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    dst = (np.arange(count) % 30).astype(np.int32)
    # 65,535 at one delay pad to 65,536; 65,534 over three delays with two odd counts to as many
    d = np.ones(count, np.int32) if D == 1 else np.where(np.arange(count) < 3, 2, np.where(np.arange(count) < 6, 3, 1)).astype(np.int32)
    net = (params, np.zeros(count, np.int32), dst, np.full(count, 1e-15, np.float32), d)
    with pytest.raises(B.BsimError) as err:
        engine(net, pop=(np.arange(n) >= 30).astype(np.int32))
    assert err.value.code == -7 and "65535" in str(err.value)
