"""fvb_read_header: the first 32 bytes of a device stream at any address, in
stream order; host memory is rejected without a launch."""

import ctypes

import numpy as np
import pytest
import torch

from fastvid_b200 import _native
from fastvid_b200.codec import header_of


@pytest.mark.gpu
@pytest.mark.parametrize("lead", (0, 1, 7, 16, 33))
def test_header_at_any_address(cuda, lead):
    data = torch.arange(200, dtype=torch.int32).mul(37).remainder(256).to(torch.uint8)
    dev = torch.zeros(200, dtype=torch.uint8, device=cuda)
    dev.copy_(data)  # on the stream that the read is ordered after
    for n in (32, 33, 100):
        view = dev[lead:lead + n]
        assert header_of(view) == bytes(data[lead:lead + 32].numpy())
    assert header_of(dev[lead:lead + 90:2]) == bytes(data[lead:lead + 64:2].numpy())  # strided: copied


def test_host_memory_is_rejected_before_any_launch():
    lib = _native.load()
    host = np.zeros(64, dtype=np.uint8)
    out = ctypes.create_string_buffer(32)
    before = lib.fvb_launch_count()
    assert lib.fvb_read_header(host.ctypes.data, out, None) == -1
    assert _native.last_error() == "encoded stream must be device memory"
    assert lib.fvb_read_header(host.ctypes.data, None, None) == -1
    assert lib.fvb_launch_count() == before
