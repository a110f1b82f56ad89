"""Scalar reset values filled in on the device are what a conversion on the host gives."""
import numpy as np
import pytest
import torch

from btorch_b200.models.base import ResetValue, _memory_var

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value,dtype", [
    (-0.1, torch.float64), (0.1, None), (np.float64(0.1), torch.float64), (np.asarray(1e300), torch.float32),
    (70000.0, torch.float16), (-70000.0, torch.float16), (0.1, torch.bfloat16), (1.7, torch.int64), (3, None),
    (True, None), (float("nan"), torch.float32), (float("-inf"), torch.float32), (torch.tensor(0.25), torch.float64),
    (torch.tensor(2.0, requires_grad=True), None)])
@pytest.mark.parametrize("batch", [None, 2, (2, 3)])
def test_device_fill_equals_host_conversion(value, dtype, batch):
    rv = ResetValue(value=value, sizes=(4,), dtype=dtype)
    want = _memory_var(rv, batch, device=torch.device("cpu"))
    got = _memory_var(rv, batch, device=torch.device("cuda"))
    assert got.dtype == want.dtype and got.shape == want.shape and got.is_cuda and not got.requires_grad
    torch.testing.assert_close(got.cpu(), want, rtol=0, atol=0, equal_nan=True)
