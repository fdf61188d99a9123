"""The predictor's MLP kernels at the edges of their 64-sample tiles, against the float64
restatement: forward, gradient and training."""
import numpy as np
import pytest

import bsim_b200 as B
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


def samples(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, 2, (n, 9)).astype(np.float32), rng.uniform(0, 2, n).astype(np.float32)


# fp32 sums of at most 64 terms per tile and of the tiles' parts: relative error of a few 2^-24
# times the square root of the number of terms
@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 64 * 148 + 1, 300000])
def test_forward_and_gradient_at_tile_edges(n):
    p = B.mlp_init(n)
    x, y = samples(n, n)
    f = mlp_oracle.forward(p, x)
    assert np.allclose(B.mlp_forward(p, x), f, rtol=1e-5, atol=1e-6)
    g, loss = B.mlp_grad(p, x, y)
    l_ref, g_ref = mlp_oracle.loss_and_grad(p, x, y)
    assert abs(loss - l_ref) <= 1e-5 * abs(l_ref)
    assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)


@pytest.mark.parametrize("n,batch", [(1, 5), (200, 64), (1000, 130), (9000, 4096)])
def test_first_training_steps(n, batch):
    """One epoch: the batches of the seeded order, each followed by an Adam step; samples past the
    last whole batch are not used."""
    x, y = samples(n, 3 * n)
    p0 = B.mlp_init(7)
    p1, loss = B.mlp_train(p0, x, y, epochs=1, batch=batch, lr=1e-3, seed=9)
    mask = (1 << 64) - 1

    def mix(v):
        v ^= v >> 30
        v = v * 0xbf58476d1ce4e5b9 & mask
        v ^= v >> 27
        v = v * 0x94d049bb133111eb & mask
        return v ^ v >> 31

    idx = list(range(n))
    for i in range(n - 1, 0, -1):  # epoch 0
        j = mix((mix(9) + i * 0xd1b54a32d192ed03 + 1) & mask) % (i + 1)
        idx[i], idx[j] = idx[j], idx[i]
    p, m, v = p0.astype(np.float64), 0.0, 0.0
    bs = min(batch, n)
    for k, b0 in enumerate(range(0, n - bs + 1, bs), 1):
        at = idx[b0:b0 + bs]
        _, g = mlp_oracle.loss_and_grad(p, x[at], y[at])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** k)) / (np.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
    # a gradient near zero may take a step of either sign (2 lr): allow for a few of 4,865
    off = np.abs(p1 - p)
    assert np.sum(off > 1e-5) <= 5 and off.max() <= 2.1e-3 * k
    l_ref, _ = mlp_oracle.loss_and_grad(p1.astype(np.float64), x, y)
    assert abs(loss - l_ref) <= 1e-5 * l_ref
