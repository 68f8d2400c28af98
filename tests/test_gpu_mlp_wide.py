"""The training step's two kernels with layers wider than a block (512 threads: several outputs per
thread, their biases by every thread), at and beside that width. Tolerances as in test_gpu_mlp.py: loss
1e-4, gradients 2e-4 of the largest."""

import numpy as np
import pytest

from oracle.mlp import loss_and_grad
from test_gpu_mlp_step import _adam, _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,n", [([1, 511, 1], 17), ([1, 512, 1], 33), ([1, 513, 1], 33), ([1, 520, 1], 49),
                                      ([2, 560, 1], 16), ([560, 1, 2], 31), ([1, 1, 540], 20)])
def test_layers_wider_than_a_block(widths, n):
    from mdelast_b200.mlp import MLP
    # parameters and gradients, padded, and the activations of 16 samples within 200 KB: two kernels
    params = sum((a + 1) * (b + 1) for a, b in zip(widths, widths[1:]))
    assert 4 * (2 * (params + 3) + 2 * 20 * (sum(widths) + max(widths))) <= 200 * 1024
    net = MLP(widths, seed=9)
    x, y = _data(widths, n)
    p = net.params.astype(np.float64)
    loss, g = net.gradients(x, y)
    lo, go = loss_and_grad(p, widths, x, y)
    assert abs(loss / lo - 1) < 1e-4
    assert np.max(np.abs(g - go)) / np.max(np.abs(go)) < 2e-4
    net.train(x, y, 3, lr=1e-4)
    q = _adam(p, widths, x, y, 3, 1e-4)
    assert np.linalg.norm(net.params - q) <= 1e-2 * np.linalg.norm(q - p)
