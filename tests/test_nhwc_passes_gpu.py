"""The passes around the convolution kernel: planes -> NHWC (chain export and the planes-out plan), the
inverse filter permutation, the bias that the last pass adds, and the staging of a strided 1x1 filter's
pixels.  The passes only move fp16 values and add one, so everything but the strided convolution is
compared bit for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle_api as oa
import shflbw_sparse_nn_b200 as sb
from conftest import assert_close_fp16
from gpu_util import dev, host, run_spconv
from shflbw_sparse_nn_b200 import _cabi
from shflbw_sparse_nn_b200.build import build_fault_inject_library
from shflbw_sparse_nn_b200.nn import ShflBWConv2d, densify

pytestmark = pytest.mark.gpu


@pytest.fixture
def flib():
    """The test build, which tells how an export is split and can split it finer."""
    lib = _cabi.load_library(build_fault_inject_library())
    lib.shflbw_debug_export_steps.argtypes, lib.shflbw_debug_export_steps.restype = [C.c_longlong, C.c_int], C.c_int
    lib.shflbw_debug_set_export_pixels.argtypes, lib.shflbw_debug_set_export_pixels.restype = [C.c_int], C.c_int
    yield lib
    lib.shflbw_debug_set_export_pixels(0)


@pytest.mark.parametrize("Bn,H,W,F,R,permute,steps", [
    (1, 1, 1, 32, 1, True, 1), (3, 5, 7, 96, 3, True, 1), (8, 9, 4, 64, 1, False, 1), (13, 6, 6, 160, 5, True, 1),
    (40, 7, 7, 2048, 1, True, 1), (256, 14, 14, 128, 3, True, 1),
    (250, 7, 7, 2048, 1, True, 3), (117, 7, 7, 1984, 3, True, 2),       # several 64-token steps per block, the last round ragged
    (61, 9, 13, 4096, 1, False, 4),
])
def test_chain_export_is_the_transpose_of_the_planes(flib, Bn, H, W, F, R, permute, steps):
    assert flib.shflbw_debug_export_steps(H * W * (-(-Bn // 8) * 8), F) == steps
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, 8, 32, 1, 0.5, permute, 3, values="uniform")
    f.transform_and_sync_device()
    Bp = -(-Bn // 8) * 8
    buf = sb.uniform_half(4, F * (H + R - 1) * (W + R - 1) * Bp).reshape(F, H + R - 1, W + R - 1, Bp)
    y = torch.full((Bn, H, W, F), float("nan"), dtype=torch.float16, device="cuda")
    sb.chain_export_nhwc(dev(buf), Bn, H, W, F, R, R, f if permute else None, y, torch.cuda.current_stream())
    torch.cuda.synchronize()
    want = np.empty((Bn, H, W, F), np.float16)
    core = buf[:, R // 2:R // 2 + H, R // 2:R // 2 + W, :Bn].transpose(3, 1, 2, 0)
    want[..., f.row_permute_ids if permute else np.arange(F)] = core
    assert np.array_equal(host(y).view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("pixels", [1, 5, 34, 35])
def test_chain_export_in_several_launches(flib, pixels):
    Bn, H, W, F, R = 13, 5, 7, 200, 3
    buf = sb.uniform_half(4, F * (H + R - 1) * (W + R - 1) * 16).reshape(F, H + R - 1, W + R - 1, 16)
    y = torch.full((Bn, H, W, F), float("nan"), dtype=torch.float16, device="cuda")
    planes = dev(buf)
    flib.shflbw_debug_set_export_pixels(pixels)
    assert flib.shflbw_chain_export_nhwc(planes.data_ptr(), Bn, H, W, F, R, R, None, y.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream) == _cabi.OK
    torch.cuda.synchronize()
    want = buf[:, 1:1 + H, 1:1 + W, :Bn].transpose(3, 1, 2, 0)
    assert np.array_equal(host(y).view(np.uint16), np.ascontiguousarray(want).view(np.uint16))


@pytest.mark.parametrize("V,F,C,R,permute", [
    (64, 192, 256, 3, True),            # planes out
    (64, 128, 64, 1, True), (32, 96, 64, 1, True), (128, 1024, 32, 1, True),    # positions out + inverse permutation (F <= 512, above)
    (32, 64, 64, 3, False), (16, 48, 64, 1, False), (128, 256, 32, 1, False),   # positions out, bias in the kernel's epilogue
])
@pytest.mark.parametrize("Bn,H", [(1, 3), (5, 11)])
def test_bias_equals_a_separate_fp16_add(V, F, C, R, permute, Bn, H):
    f = sb.BlockwiseSpFilter().init_random(F, R, R, C, V, 1, 0.3, permute, 21, values="uniform")
    bias = dev(sb.uniform_half(22, F))
    conv = ShflBWConv2d(f, 1, bias).cuda()
    x = dev(sb.uniform_half(23, Bn * H * H * C).reshape(Bn, H, H, C)).permute(0, 3, 1, 2)
    y = conv(x)
    conv.bias = None
    want = conv(x).permute(0, 2, 3, 1) + bias
    misaligned = torch.zeros(F + 1, dtype=torch.float16, device="cuda")[1:]
    misaligned.copy_(bias)
    conv.bias = misaligned              # added by torch
    y2 = conv(x)
    torch.cuda.synchronize()
    f.device_status()
    assert torch.equal(y.permute(0, 2, 3, 1), want) and torch.equal(y, y2)
    if V == 32 and permute:
        ref = oa.spconv_ref_nhwc(Bn, H, H, C, F, R, R, 1, V, f.indptr, f.indices, f.values, f.row_permute_ids,
                                 host(x.permute(0, 2, 3, 1).contiguous())) + host(bias).astype(np.float32)
        assert_close_fp16(host(y.permute(0, 2, 3, 1).contiguous()), ref, abs_=2e-3, what="bias vs oracle")


@pytest.mark.parametrize("Bn,H,W,stride,V,C", [(1, 1, 1, 2, 32, 8), (3, 27, 26, 2, 32, 72), (9, 10, 13, 3, 64, 64), (2, 8, 8, 9, 128, 64)])
def test_strided_1x1_filters_stage_only_the_pixels_they_visit(Bn, H, W, stride, V, C):
    f = sb.BlockwiseSpFilter().init_random(2 * V, 1, 1, C, V, 1, 0.4, True, 31, values="uniform")
    x = sb.uniform_half(32, Bn * H * W * C).reshape(Bn, H, W, C)
    y, _ = run_spconv(f, Bn, H, W, stride, x)
    sub, _ = run_spconv(f, Bn, -(-H // stride), -(-W // stride), 1, np.ascontiguousarray(x[:, ::stride, ::stride]))
    assert np.array_equal(y.view(np.uint16), sub.view(np.uint16))
    ref = oa.spconv_ref_nhwc(Bn, H, W, C, 2 * V, 1, 1, stride, V, f.indptr, f.indices, f.values, f.row_permute_ids, x)
    assert_close_fp16(y, ref, what="strided 1x1 vs oracle")


@pytest.mark.parametrize("V,C,R,Bn,H", [
    (64, 24, 3, 1, 4), (64, 24, 3, 9, 5), (128, 24, 3, 2, 5),      # 216 columns a block; images beyond the batch, 128-token tiles
    (128, 24, 3, 16, 14),                                          # an output of 146 MB
    (64, 24, 1, 3, 4),                                             # 24 columns
])
def test_more_filters_than_the_inverse_permutation_holds(V, C, R, Bn, H):
    F = 23296                                                      # that pass: 10 F bytes of shared memory, 23 244 filters
    f = sb.BlockwiseSpFilter().init_random(F, R, R, C, V, 1, 1.0, True, 33, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(34, Bn * H * H * C).reshape(Bn, H, H, C))
    y = torch.full((Bn, H, H, F), float("nan"), dtype=torch.float16, device="cuda")
    sb.SpconvBlockwiseOp().initialize(f, Bn, H, H, 1, x, y)(torch.cuda.current_stream())
    torch.cuda.synchronize()
    f.device_status()
    w = torch.from_numpy(densify(f)).cuda().double()
    halo = torch.nn.functional.pad(x.double(), (0, 0, R // 2, R // 2, R // 2, R // 2))
    cols = torch.cat([halo[:, r:r + H, s:s + H] for r in range(R) for s in range(R)], 3).reshape(-1, R * R * C)
    want, size = cols @ w.t(), cols.abs() @ w.abs().t()
    # 32-bit sums of n products in any order, n * 2^-23 * sum |a b| (sums chopped, not rounded), and a rounding to fp16
    assert ((y.reshape(-1, F).double() - want).abs() <= R * R * C * 2.0 ** -23 * size + want.abs() * 2.0 ** -11 + 2.0 ** -25).all()


def test_filters_of_few_rows_a_block_keep_that_limit():
    for Bn in (1, 64):                                             # no planes for 32 rows: refused for every size
        f = sb.BlockwiseSpFilter().init_random(23296, 1, 1, 8, 32, 1, 1.0, True, 35, values="uniform")
        f.transform_and_sync_device()
        x, y = (torch.zeros(Bn * 16 * n, dtype=torch.float16, device="cuda") for n in (8, 23296))
        with pytest.raises(sb.ShflbwError) as e:
            sb.SpconvBlockwiseOp().initialize(f, Bn, 4, 4, 1, x, y)
        assert e.value.status == _cabi.ERR_UNSUPPORTED
