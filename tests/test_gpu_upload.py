"""Uploads that do not wait: the kernels queued behind them read the caller's values,
whatever the caller does with its array afterwards, on the default and on another stream."""

import numpy as np
import pytest
import torch

from ssms_b200 import _device as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 129, 100_000])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float64])
def test_upload_keeps_the_values_of_the_call(cuda, n, dtype):
    busy = torch.ones(64 << 20, device="cuda")
    for k in range(4):
        x = (np.arange(n) * (k + 1)).astype(dtype)
        busy.mul_(1.0)  # the copy queues behind this
        t = D.upload(x)
        twice = t + t
        x[:] = -1
        np.testing.assert_array_equal(twice.cpu().numpy(), (2 * (np.arange(n) * (k + 1))).astype(dtype))
    s = torch.cuda.Stream()
    x = np.arange(n).astype(dtype)
    busy.mul_(1.0)
    t = D.upload(x, s)
    with torch.cuda.stream(s):
        np.testing.assert_array_equal((t + t).cpu().numpy(), 2 * x)
