"""Once a block of the batch kernel has given up at the grid barrier, the others leave it without polling to their limit."""
import ctypes as C

import pytest
import torch

from xadvcool_b200 import _capi
from xadvcool_b200._tensors import stream_ptr

pytestmark = pytest.mark.gpu


def test_barrier_ends_soon_after_an_error(cuda):
    s, ms = stream_ptr(torch.device("cuda")), C.c_float()
    _capi.call("xac_test_barrier_after_error", 1, C.byref(ms), s)  # the kernel's first launch
    _capi.call("xac_test_barrier_after_error", 1 << 20, C.byref(ms), s)
    # 2^20 polls sleep 32 ns each, 30 ms and more; the error is looked at every 1024 polls
    assert ms.value < 10.0
