"""Setting a network's parameters, and creating one, is complete before its first training step,
whatever else keeps the device's legacy stream busy: training afterwards gives the bits it gives on
a quiet device. The network's kernels run on a stream of its own that does not wait for the legacy
one, so a reset issued there could land after the steps that follow it."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _BusyLegacyStream:
    """Short kernels on the legacy stream from another thread, a few milliseconds in flight."""

    def __enter__(self):
        import torch
        self._stop, ready = threading.Event(), threading.Event()

        def work():
            a = torch.ones(2048, 2048, device="cuda")
            while not self._stop.is_set():
                for _ in range(20):
                    a @ a
                ready.set()
                torch.cuda.default_stream().synchronize()
        self._thread = threading.Thread(target=work)
        self._thread.start()
        ready.wait(60)

    def __exit__(self, *exc):
        self._stop.set()
        self._thread.join()


# two kernels per step, and layer by layer
@pytest.mark.parametrize("widths", [[2, 64, 64, 64, 4], [2, 256, 256, 4]])
def test_reset_comes_before_training(widths):
    from mdelast_b200.mlp import MLP
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (300, 2)).astype(np.float32)
    y = rng.uniform(-1, 1, (300, 4)).astype(np.float32)

    def fresh():
        net = MLP(widths, seed=7)
        net.train(x, y, 3, lr=1e-2)
        return net.params

    net = MLP(widths, seed=7)
    start = net.params
    net.train(x, y, 3, lr=1e-2)
    want = net.params
    with _BusyLegacyStream():
        for _ in range(10):
            net.params = start
            net.train(x, y, 3, lr=1e-2)
            assert np.array_equal(net.params, want)
            assert np.array_equal(fresh(), want)
