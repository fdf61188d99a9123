"""Pushed cycles with few spikes, one launch per cycle: rows that are cut among warps and rows that are
not, against the oracle."""
import numpy as np
import pytest

import bsim_b200 as B
from test_gpu_loop import network, reference, same

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)


@pytest.mark.parametrize("n,D,degree", [(400, 1, 383), (400, 1, 384), (60, 1, 9001), (300, 2, 1501), (7, 3, 2049)])
def test_rows_around_the_cut(n, D, degree):
    net = network(n, D, degree, seed=degree)
    net[3][:] *= np.float32(20.0 / degree)
    steps = 80
    eng = B.Engine.from_arrays(*net, DT, opts=B.options(block_threads=512))
    eng.record(steps, n * steps)
    eng.run(steps)
    assert eng.info().many_cycles == 0
    ref = reference(net, steps, eng)
    assert ref["fire_count"].sum() > 0 and np.median(ref["spikes_per_step"]) < 1000
    same(eng, ref, steps)
    eng.close()
