"""What the operators take for a buffer or a stream: an integer, or an object that tells one, of whatever
integer type it is (ctypes itself takes only Python's)."""
import ctypes as C

import numpy as np
import pytest
import torch

from shflbw_sparse_nn_b200 import blockwise as bw


class Holder:
    def __init__(self, value):
        self.cuda_stream, self.data_ptr = value, lambda: value


@pytest.mark.parametrize("value", [4096, np.int64(4096), np.uint64(4096), torch.tensor(4096).numpy()[()]])
def test_addresses_of_any_integer_type(value):
    for f in (bw._ptr, bw._stream_ptr):
        for x in (value, Holder(value)):
            assert C.c_void_p(f(x)).value == 4096
        assert f(None) is None
