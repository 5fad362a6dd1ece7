"""A call whose kernel cannot be set up launches nothing.  The failure is made on the host, in the test
build of the library: the opt-in to a kernel's shared memory is refused."""
import ctypes as C

import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from gpu_util import dev
from shflbw_sparse_nn_b200 import _cabi
from shflbw_sparse_nn_b200.build import build_fault_inject_library

pytestmark = pytest.mark.gpu


@pytest.fixture
def flib():
    lib = _cabi.load_library(build_fault_inject_library())
    lib.shflbw_debug_fail_set_up_after.restype = C.c_int
    lib.shflbw_debug_fail_set_up_after.argtypes = [C.c_int]
    yield lib
    lib.shflbw_debug_fail_set_up_after(-1)


def _poison(n):
    return torch.full((n,), 7.0, dtype=torch.float16, device="cuda")


def test_biased_convolution_launches_nothing(flib):
    h = C.c_void_p()
    assert flib.shflbw_filter_create_random(96, 1, 1, 32, 32, 1, 0.5, 0, 3, _cabi.VALUES_UNIFORM, C.byref(h)) == _cabi.OK
    try:
        assert flib.shflbw_matrix_to_device(h) == _cabi.OK
        x, out, bias = dev(sb.uniform_half(4, 8 * 25 * 32)), _poison(8 * 25 * 96), _poison(96)
        st = _cabi.SpconvState()
        assert flib.shflbw_spconv_init(h, 8, 5, 5, 1, x.data_ptr(), out.data_ptr(), 1.0, _cabi.KERNEL_AUTO, C.byref(st)) == _cabi.OK
        staged = _poison(32 * 25 * 8)                      # in place of the filter's own scratch: watched here
        st.staged_in = staged.data_ptr()
        stream = torch.cuda.current_stream().cuda_stream
        flib.shflbw_debug_fail_set_up_after(0)
        assert flib.shflbw_spconv_exec_bias(C.byref(st), bias.data_ptr(), stream) == _cabi.ERR_CUDA
        torch.cuda.synchronize()
        assert (staged == 7).all() and (out == 7).all()
        flib.shflbw_debug_fail_set_up_after(-1)
        assert flib.shflbw_spconv_exec_bias(C.byref(st), bias.data_ptr(), stream) == _cabi.OK
        torch.cuda.synchronize()
        assert flib.shflbw_matrix_device_status(h) == _cabi.OK and not (staged == 7).any()
    finally:
        flib.shflbw_matrix_destroy(h)


def test_biased_linear_layer_launches_nothing(flib):
    h = C.c_void_p()
    assert flib.shflbw_matrix_create_random(256, 128, 64, 1, 0.5, 1, 3, _cabi.VALUES_UNIFORM, C.byref(h)) == _cabi.OK
    try:
        assert flib.shflbw_matrix_to_device(h) == _cabi.OK
        x, xt, out, bias = dev(sb.uniform_half(4, 24 * 128)), _poison(24 * 128), _poison(24 * 256), _poison(256)
        stream = torch.cuda.current_stream().cuda_stream
        args = (h, 24, x.data_ptr(), bias.data_ptr(), xt.data_ptr(), 24, out.data_ptr(), stream)
        flib.shflbw_debug_fail_set_up_after(1)           # the plain kernel at init, not the biased one
        assert flib.shflbw_linear_exec(*args) == _cabi.ERR_CUDA
        torch.cuda.synchronize()
        assert (xt == 7).all() and (out == 7).all()
        flib.shflbw_debug_fail_set_up_after(-1)
        assert flib.shflbw_linear_exec(*args) == _cabi.OK
        torch.cuda.synchronize()
        assert flib.shflbw_matrix_device_status(h) == _cabi.OK and not (xt == 7).any()
    finally:
        flib.shflbw_matrix_destroy(h)
