"""Several host threads on one engine: reads while another thread runs it are of one moment each."""
import hashlib
import threading
import time

import numpy as np
import pytest

import bsim_b200 as B

pytestmark = pytest.mark.gpu
DT = np.float32(1e-4)
LIF = [-0.065, -0.065, -0.065, 0.25e-9, 20e-3, 2e-3, 5e-3, 10e-3, -0.050, 0.0]
FIELDS = ("v", "i_E", "i_I", "refrac")


def engine(n):
    rng = np.random.default_rng(7)
    params = np.tile(np.array(LIF, np.float32), (n, 1))
    params[:, 0] = rng.uniform(-0.065, -0.051, n)
    params[:, 9] = rng.uniform(1e-9, 8e-9, n)
    src, dst = rng.integers(0, n, 3 * n).astype(np.int32), rng.integers(0, n, 3 * n).astype(np.int32)
    return B.Engine.from_arrays(params, src, dst, rng.uniform(-2e-10, 3e-10, 3 * n).astype(np.float32),
                                rng.integers(1, 6, 3 * n).astype(np.int32), DT)


def digest(arrays):
    return hashlib.sha1(b"".join(np.ascontiguousarray(a).tobytes() for a in arrays)).digest()


@pytest.mark.parametrize("n", [9000, 60000])  # many cycles per launch and one; both read through page-locked memory
def test_reads_while_another_thread_runs(n):
    steps = 150
    ref = engine(n)
    states, counts = set(), set()
    for k in range(steps + 1):
        st = ref.state()
        states.add(digest(st[f] for f in FIELDS))
        counts.add(digest([ref.fire_count()]))
        ref.run(1)
    ref.close()
    assert len(states) == steps + 1 and len(counts) > steps // 2
    eng = engine(n)
    done = threading.Event()
    seen, errors = [], []

    def reader():
        try:
            while not done.is_set():
                st = eng.state()
                c = eng.fire_count()
                seen.append((digest(st[f] for f in FIELDS), digest([c])))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=reader) for _ in range(3)]
    eng.state()
    for t in threads:
        t.start()
    for k in range(steps):
        eng.run(1)
        while len(seen) < k // 5 and not errors:  # the readers keep up
            time.sleep(1e-4)
    done.set()
    for t in threads:
        t.join()
    eng.close()
    assert not errors and len(seen) > 20
    assert all(s in states for s, _ in seen)
    assert all(c in counts for _, c in seen)
