"""The sixteen-epilogue-warp kernel copies the addend of an item (a chained layer's residual, or C)
to shared memory an item ahead.  It performs the arithmetic of the eight-warp kernel in the same
order, so the two must agree bit for bit: with several items per block, with one item only for some
of the blocks, with a ragged last token tile, with a halo around the output planes, with a plane map
and with the residual added in place."""
import ctypes as C

import numpy as np
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from shflbw_sparse_nn_b200 import _cabi
from gpu_util import dev, epilogue_warps, host, operand_swap, run_spmm, tile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Bn,H,R_next,mapped,in_place", [
    (8, 16, 1, True, False),        # 8 token tiles x 4 blocks: at most one item per block
    (40, 33, 1, True, False),       # several items per block, ragged last tile
    (40, 33, 3, False, False),      # output with a halo
    (64, 24, 1, False, True),       # out = relu(conv + out)
])
def test_chained_residual_matches_the_eight_warp_kernel(Bn, H, R_next, mapped, in_place):
    Cc, F = 64, 256
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, Cc, 64, 1, 0.3, True, 5, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(6, sb.chain_buffer_elems(Cc, H, H, Bn, 1, 1)))
    n_out = sb.chain_buffer_elems(F, H, H, Bn, R_next, R_next)
    res = dev(sb.uniform_half(7, n_out))
    got = {}
    for ew in (8, 16):
        out = res.clone() if in_place else torch.zeros(n_out, dtype=torch.float16, device="cuda")
        with operand_swap(0), epilogue_warps(ew), tile(256):
            op = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, x, out, R_next, R_next, alpha=0.5, relu=True)
            op.set_residual(out if in_place else res, None if mapped else "same")
        assert op._state.variant == (2 if ew == 16 else 0)
        op(torch.cuda.current_stream())
        torch.cuda.synchronize()
        f.device_status()
        got[ew] = host(out).view(np.uint16)
    assert np.array_equal(got[8], got[16])


def test_residual_picks_the_sixteen_warp_kernel_for_two_stages_of_columns():
    Cc, F, Bn, H = 512, 512, 64, 20           # 102 of 512 columns, padded to 112 a block; 800 items
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, Cc, 64, 1, 0.2, True, 8, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(9, sb.chain_buffer_elems(Cc, H, H, Bn, 1, 1)))
    n_out = sb.chain_buffer_elems(F, H, H, Bn, 1, 1)
    res = dev(sb.uniform_half(10, n_out))
    got = []
    for force in (None, 8):
        out = torch.zeros(n_out, dtype=torch.float16, device="cuda")
        with epilogue_warps(force):
            op = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, x, out, 1, 1)
            assert op._state.variant == 0
            op.set_residual(res, None)
        assert op._state.variant == (0 if force else 2)
        op(torch.cuda.current_stream())
        torch.cuda.synchronize()
        f.device_status()
        got.append(host(out).view(np.uint16))
    assert np.array_equal(got[0], got[1])


def test_refused_residual_leaves_the_state_as_it_was():
    Cc, F, Bn, H = 512, 512, 64, 20           # a residual would switch to the sixteen-warp kernel
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, Cc, 64, 1, 0.2, True, 8, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(9, sb.chain_buffer_elems(Cc, H, H, Bn, 1, 1)))
    out = torch.zeros(sb.chain_buffer_elems(F, H, H, Bn, 1, 1), dtype=torch.float16, device="cuda")
    op = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, x, out, 1, 1)
    before = bytes(op._state)
    bad = np.arange(F, dtype=np.int32)
    for value in (-1, F):
        bad[-1] = value
        rc = _cabi.lib().shflbw_spconv_chain_set_residual(f._h, C.byref(op._state), out.data_ptr(), bad.ctypes.data)
        assert rc == _cabi.ERR_BAD_FORMAT and bytes(op._state) == before
    bad[-1] = F - 1
    assert _cabi.lib().shflbw_spconv_chain_set_residual(f._h, C.byref(op._state), out.data_ptr(), bad.ctypes.data) == 0
    assert op._state.variant == 2 and op._state.residual == out.data_ptr() and op._state.residual_map


@pytest.mark.parametrize("Cc,padded_cols,ring", [(64, 112, 6), (80, 128, 6), (88, 144, 8), (200, 272, 8)])
def test_ring_of_the_sixteen_warp_kernel(Cc, padded_cols, ring):
    """Eight stages where nothing is added and a block takes two of them, six with slots for an addend
    otherwise; a residual bound later moves a layer to the six.  Same bits as the eight-warp kernel."""
    F, Bn, H = 256, 40, 33
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, Cc, 64, 1, 0.3, True, 5, values="uniform")
    f.transform_and_sync_device()
    assert sum(-(-np.diff(f.indptr) // 16) * 16) == padded_cols        # of four blocks
    x = dev(sb.uniform_half(6, sb.chain_buffer_elems(Cc, H, H, Bn, 1, 1)))
    n_out = sb.chain_buffer_elems(F, H, H, Bn, 1, 1)
    res = dev(sb.uniform_half(7, n_out))
    got = {}
    for ew in (8, 16):
        out = torch.zeros(n_out, dtype=torch.float16, device="cuda")
        with operand_swap(0), epilogue_warps(ew), tile(256):
            op = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, x, out, 1, 1, relu=True)
        if ew == 16:
            assert (op._state.variant, op._state.stages) == (2, ring)
        op(torch.cuda.current_stream())
        plain = out.clone()
        op.set_residual(res)
        if ew == 16:
            assert (op._state.variant, op._state.stages) == (2, 6)
        op(torch.cuda.current_stream())
        torch.cuda.synchronize()
        f.device_status()
        got[ew] = host(plain).view(np.uint16), host(out).view(np.uint16)
    assert np.array_equal(got[8][0], got[16][0]) and np.array_equal(got[8][1], got[16][1])
    assert not np.array_equal(got[16][0], got[16][1])


@pytest.mark.parametrize("N", [256 * 37, 256 * 80 + 24])
def test_spmm_without_an_addend_matches_the_eight_warp_kernel(N):
    m = sb.BlockwiseSpMatrix().init_random(512, 200, 64, 1, 0.2, True, 11, values="uniform")
    B = sb.uniform_half(12, m.ncol * N).reshape(m.ncol, N)
    got = []
    for ew, stages in ((8, None), (16, 8)):
        with operand_swap(0), epilogue_warps(ew):
            y, op = run_spmm(m, N, B, alpha=0.5, tokens=256)
        assert op._state.variant == (2 if ew == 16 else 0) and stages in (None, op._state.stages)
        got.append(y.view(np.uint16))
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("N", [256 * 37, 256 * 80 + 24])
def test_spmm_beta_matches_the_eight_warp_kernel(N):
    m = sb.BlockwiseSpMatrix().init_random(512, 200, 64, 1, 0.2, True, 11, values="uniform")
    B = sb.uniform_half(12, 200 * N).reshape(200, N)
    Cm = sb.uniform_half(13, 512 * N).reshape(512, N)
    out = []
    for ew in (8, 16):
        with operand_swap(0), epilogue_warps(ew):
            D, op = run_spmm(m, N, B, alpha=0.5, Cm=Cm, beta=0.75, tokens=256)
        assert op._state.variant == (2 if ew == 16 else 0)
        out.append(D.view(np.uint16))
    assert np.array_equal(out[0], out[1])
