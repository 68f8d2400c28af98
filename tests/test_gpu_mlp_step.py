"""The training step's two kernels against the float64 oracle at the edges of their sample
tiles (16 samples, 148 blocks) and layer widths (odd, wider than a block), and next to a network
too large for them. Tolerances as in test_gpu_mlp.py: loss 1e-4, gradients 2e-4 of the largest."""

import numpy as np
import pytest

from oracle.mlp import forward, loss_and_grad

pytestmark = pytest.mark.gpu


def _data(widths, n, seed=4):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, (n, widths[0])).astype(np.float32)
    y = np.sin(x @ rng.normal(size=(widths[0], widths[-1]))).astype(np.float32)
    return x, y


def _adam(p, widths, x, y, steps, lr):
    m1, m2 = np.zeros_like(p), np.zeros_like(p)
    for k in range(1, steps + 1):
        _, g = loss_and_grad(p, widths, x, y)
        m1 = 0.9 * m1 + 0.1 * g
        m2 = 0.999 * m2 + 0.001 * g * g
        p = p - lr * (m1 / (1 - 0.9 ** k)) / (np.sqrt(m2 / (1 - 0.999 ** k)) + 1e-8)
    return p


@pytest.mark.parametrize("widths,n", [([2, 64, 64, 64, 4], 1), ([2, 64, 64, 64, 4], 15),
                                      ([3, 64, 64, 64, 4], 17), ([2, 64, 64, 64, 4], 148 * 16 + 3),
                                      ([5, 7, 33, 3], 130), ([4, 2], 50), ([3, 300, 4], 40),
                                      ([2, 16, 16, 16, 16, 16, 16, 16, 1], 97),
                                      ([2, 256, 256, 4], 33)])
def test_step_matches_oracle(widths, n):
    from mdelast_b200.mlp import MLP
    net = MLP(widths, seed=9)
    x, y = _data(widths, n)
    p = net.params.astype(np.float64)
    loss, g = net.gradients(x, y)
    lo, go = loss_and_grad(p, widths, x, y)
    assert abs(loss / lo - 1) < 1e-4
    assert np.max(np.abs(g - go)) / np.max(np.abs(go)) < 2e-4
    # three steps move the parameters by about 3 lr; Adam's early steps keep a gradient's sign and
    # lose its size, so entries far below the others may differ by a step: compare the network
    last = net.train(x, y, 3, lr=1e-4)
    q = _adam(p, widths, x, y, 3, 1e-4)
    assert np.linalg.norm(net.params - q) <= 1e-2 * np.linalg.norm(q - p)
    assert np.allclose(net(x), forward(net.params.astype(np.float64), widths, x), rtol=1e-4, atol=1e-5)
    assert abs(last / loss_and_grad(net.params.astype(np.float64), widths, x, y)[0] - 1) < 1e-3
