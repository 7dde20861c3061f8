"""The asynchronous energy call on streams that do not wait for the default stream."""
import ctypes

import numpy as np
import pytest

import cgppd_gb300
from helpers import device_array, ptr
from test_dropin_gpu import L, eon, synthetic_packed  # noqa: F401  (L: fixture)

pytestmark = pytest.mark.gpu


def test_first_call_on_a_stream_behind_a_busy_default_stream(L):  # noqa: F811
    """A stream's scratch is set up by its first call, and again by a larger one."""
    import torch
    rng = np.random.default_rng(4)
    calls = []
    for nmol in (4, 30):  # 10 and some 800 CTAs
        pos, meta = synthetic_packed(rng, nmol, [90, 140], 200.0)
        calls.append((device_array(pos), device_array(meta), pos.shape[0], eon(L, pos, meta, 200.0)))
    out = torch.zeros(1, device="cuda")
    stream = torch.cuda.Stream()
    for dp, dm, n, want in calls:
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream
        for _ in range(3):
            L.CUDA_EonDevice_async(ptr(dp), ptr(dm), None, None, None, None, ptr(out), 1, 32, n, 0,
                                   ctypes.c_void_p(stream.cuda_stream))
        stream.synchronize()
        cgppd_gb300.check("EonDevice_async")
        torch.cuda.synchronize()
        # (one rounding to FP32; float-float sums, in whatever order, are far below it)
        assert abs(float(out[0]) - want) <= 2.0 ** -23 * abs(want) + 1e-9
