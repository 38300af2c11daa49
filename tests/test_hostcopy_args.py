"""Context.copy_to_device and copy_to_host refuse what they could not copy
within the tensor (before the library is called: no GPU is needed)."""

import numpy as np
import pytest
import torch

import polariseq_b200 as pq


@pytest.mark.parametrize("tensor,array,offset", [
    (torch.empty(10), np.empty(11, np.float32), 0),             # longer than the tensor
    (torch.empty(10), np.empty(10, np.float32), 4),             # past its end
    (torch.empty(10), np.empty(4, np.float32), -4),             # before its start
    (torch.empty(10, dtype=torch.int32), np.empty(6), 0),       # 48 bytes of doubles
    (torch.empty(10, 10), np.empty((10, 10), np.float32).T, 0),
    (torch.empty(10, 10), np.empty(20, np.float32)[::2], 0),
    (torch.empty(10, 10).t(), np.empty(20, np.float32), 0)])
def test_copies_outside_the_tensor_are_refused(tensor, array, offset):
    ctx = pq.Context.__new__(pq.Context)  # (no device behind it)
    with pytest.raises(ValueError):
        ctx.copy_to_device(tensor, array, offset)
    if offset == 0:
        with pytest.raises(ValueError):
            ctx.copy_to_host(array, tensor)
