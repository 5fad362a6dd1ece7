"""Residuals that the copy engine fetches in boxes of 64 tokens (sixteen epilogue warps): the arithmetic of the kernel that
copies them by cp.async, in the same order, so the two agree bit for bit.  Sizes: fewer chunks than slots, several laps of
them, a last box that the tensor ends in, an output with a halo, blocks without columns, special values, in place."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from gpu_util import dev, epilogue_warps, host, operand_swap, tile
from shflbw_sparse_nn_b200 import _cabi
from shflbw_sparse_nn_b200.build import build_fault_inject_library

pytestmark = pytest.mark.gpu


def _layer(f, x, out, res, Bn, H, R_next, producer, relu=True):
    with operand_swap(0), epilogue_warps(16), tile(256):
        op = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, x, out, R_next, R_next, alpha=0.5, relu=relu)
        op.set_residual(res, producer)
    return op


@pytest.mark.parametrize("Bn,H,R_next,F,density,mapped,in_place,fits", [
    (8, 5, 1, 64, 0.3, True, False, True),        # 200 tokens: one item, whose last box is half beyond the tensor
    (3, 1, 1, 128, 0.3, False, False, True),      # 8 tokens
    (8, 16, 1, 256, 0.3, True, False, True),      # an item or none per block
    (61, 33, 1, 256, 0.3, True, False, True),     # eight items per block and a ragged last tile
    (64, 24, 3, 192, 0.3, True, False, True),     # halo, rows of whole boxes
    (8, 24, 3, 192, 0.3, True, False, True),
    (64, 24, 1, 256, 0.3, False, True, True),     # out = relu(conv + out)
    (40, 28, 1, 320, 0.015, True, False, True),   # some blocks without a column
    (8, 9, 3, 64, 0.3, True, False, False),       # rows of 72 tokens beside a halo: no boxes
])
def test_box_residual_equals_cp_async_residual(Bn, H, R_next, F, density, mapped, in_place, fits, monkeypatch):
    Cc = 64
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, Cc, 64, 1, density, True, 5, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(6, sb.chain_buffer_elems(Cc, H, H, Bn, 1, 1)))
    n_out = sb.chain_buffer_elems(F, H, H, Bn, R_next, R_next)
    r = sb.uniform_half(7, n_out)
    r[::97], r[1::193], r[2::389] = np.inf, np.nan, -np.inf
    res = dev(r)
    got = {}
    for box in ("0", "1"):
        monkeypatch.setenv("SHFLBW_BOX", box)
        out = res.clone() if in_place else torch.zeros(n_out, dtype=torch.float16, device="cuda")
        op = _layer(f, x, out, out if in_place else res, Bn, H, R_next, None if mapped else "same", relu=density > 0.1)
        assert (op._state.variant, op._state.box_res) == (2, int(box == "1" and fits))
        for _ in range(1 if in_place else 2):
            op(torch.cuda.current_stream())
        torch.cuda.synchronize()
        f.device_status()
        got[box] = host(out).view(np.uint16)
    assert np.array_equal(got["0"], got["1"])


def test_exchanged_and_removed_residuals_are_followed(monkeypatch):
    monkeypatch.setenv("SHFLBW_BOX", "1")
    Bn, H, F = 64, 24, 256
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, 64, 64, 1, 0.3, True, 5, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(6, sb.chain_buffer_elems(64, H, H, Bn, 1, 1)))
    n = sb.chain_buffer_elems(F, H, H, Bn, 1, 1)
    r1, r2 = dev(sb.uniform_half(7, n)), dev(sb.uniform_half(8, n))
    s = torch.cuda.current_stream()

    def run(op, out):
        op(s)
        torch.cuda.synchronize()
        f.device_status()
        return host(out).view(np.uint16).copy()

    out = torch.zeros(n, dtype=torch.float16, device="cuda")
    op = _layer(f, x, out, r1, Bn, H, 1, None)
    want = _layer(f, x, out, r2, Bn, H, 1, None)
    assert op._state.box_res == want._state.box_res == 1
    first, second = run(op, out), run(want, out)
    op._state.residual = r2.data_ptr()
    assert np.array_equal(run(op, out), second) and not np.array_equal(first, second)
    op._state.residual = None
    with operand_swap(0), epilogue_warps(16), tile(256):
        plain = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, x, out, 1, 1, alpha=0.5, relu=True)
    assert np.array_equal(run(op, out), run(plain, out))


def test_wait_limit_runs_out_beside_a_box_residual(monkeypatch):
    monkeypatch.setenv("SHFLBW_SWAP", "0")
    monkeypatch.setenv("SHFLBW_EPILOGUE_WARPS", "16")
    monkeypatch.setenv("SHFLBW_TILE", "256")
    monkeypatch.setenv("SHFLBW_BOX", "1")
    flib = _cabi.load_library(build_fault_inject_library())
    flib.shflbw_debug_withhold_arrivals_from.restype = C.c_int
    flib.shflbw_debug_withhold_arrivals_from.argtypes = [C.c_int]
    Bn, H, Cc, F = 64, 40, 64, 256
    h = C.c_void_p()
    assert flib.shflbw_filter_create_random(F, 1, 1, Cc, 64, 1, 0.3, 1, 5, _cabi.VALUES_UNIFORM, C.byref(h)) == _cabi.OK
    try:
        assert flib.shflbw_matrix_to_device(h) == _cabi.OK
        x = dev(sb.uniform_half(6, sb.chain_buffer_elems(Cc, H, H, Bn, 1, 1)))
        n = sb.chain_buffer_elems(F, H, H, Bn, 1, 1)
        res, out = dev(sb.uniform_half(7, n)), torch.zeros(n, dtype=torch.float16, device="cuda")
        st = _cabi.SpconvState()
        assert flib.shflbw_spconv_chain_init(h, Bn, H, H, 1, x.data_ptr(), out.data_ptr(), 1, 1, 0.5, 1, C.byref(st)) == _cabi.OK
        assert flib.shflbw_spconv_chain_set_residual(h, C.byref(st), res.data_ptr(), None) == _cabi.OK
        assert (st.variant, st.box_res) == (2, 1)
        stream = torch.cuda.current_stream().cuda_stream

        def launch():
            assert flib.shflbw_spconv_exec(C.byref(st), stream) == _cabi.OK
            torch.cuda.synchronize()

        launch()
        assert flib.shflbw_matrix_device_status(h) == _cabi.OK
        good = host(out).copy()
        flib.shflbw_set_wait_limit_cycles(2_000_000)
        flib.shflbw_debug_withhold_arrivals_from(5)
        t0 = time.perf_counter()
        launch()
        assert time.perf_counter() - t0 < 2.0
        assert flib.shflbw_matrix_device_status(h) == _cabi.ERR_DEVICE_TIMEOUT
        flib.shflbw_debug_withhold_arrivals_from(-1)
        flib.shflbw_set_wait_limit_cycles(400_000_000)
        out.zero_()
        launch()
        assert flib.shflbw_matrix_device_status(h) == _cabi.OK
        assert np.array_equal(host(out).view(np.uint16), good.view(np.uint16))
    finally:
        flib.shflbw_debug_withhold_arrivals_from(-1)
        flib.shflbw_set_wait_limit_cycles(400_000_000)
        flib.shflbw_matrix_destroy(h)
