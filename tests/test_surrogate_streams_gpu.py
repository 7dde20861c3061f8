"""The surrogate beside other work on the GPU: its results do not depend on what else the
device is doing."""
import numpy as np
import pytest
import torch

from cgppd_gb300 import surrogate as sg
from test_surrogate_gpu import pose_like

pytestmark = pytest.mark.gpu


def test_gradient_while_memory_is_busy():
    """Every tile image that the backward pass leaves in memory is copied while later layers
    already write shared memory; with the way to memory backed up by large copies the
    gradient is still the idle device's, bit for bit."""
    s = sg.Surrogate(batch=8192, seed=5)
    rng = np.random.default_rng(6)
    X, y = pose_like(rng, 8192), rng.normal(size=8192).astype(np.float32)
    loss, g = s.loss_grad(X, y)
    src = torch.ones(1 << 28, device="cuda")
    dst = torch.empty_like(src)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(8):
        with torch.cuda.stream(side):
            for _ in range(8):  # 2 GB each
                dst.copy_(src)
        for _ in range(4):
            lb, gb = s.loss_grad(X, y)
            assert lb == loss and np.array_equal(g, gb)
        side.synchronize()
    s.close()


def test_created_behind_a_busy_default_stream():
    """The set-up clears and fills buffers while the default stream still has work to do."""
    rng = np.random.default_rng(7)
    X, y = pose_like(rng, 256), rng.normal(size=256).astype(np.float32)
    s = sg.Surrogate(batch=256, seed=21)
    want = s.params, s.predict(X), *s.loss_grad(X, y)
    s.close()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream
    s = sg.Surrogate(batch=256, seed=21)
    got = s.predict(X), *s.loss_grad(X, y)
    torch.cuda.synchronize()
    for a, b in zip(want, (s.params, *got)):
        assert np.array_equal(a, b)
    s.close()
