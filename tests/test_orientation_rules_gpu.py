"""Which kernel a layer takes by its depth, height and size: either orientation and either gather add the same columns in the
same order, so that every choice gives the bits of the others."""
import numpy as np
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from gpu_util import dev, host, operand_swap, run_spmm
from shflbw_sparse_nn_b200 import _cabi

pytestmark = pytest.mark.gpu


def _chained(f, Bn, H, R, stride, R_next, residual, swap, gather, monkeypatch):
    if gather is None:
        monkeypatch.delenv("SHFLBW_GATHER", raising=False)
    else:
        monkeypatch.setenv("SHFLBW_GATHER", str(gather))
    Ho = -(-H // stride)
    x = dev(sb.uniform_half(3, sb.chain_buffer_elems(f.C, H, H, Bn, R, R)))
    n = sb.chain_buffer_elems(f.F, Ho, Ho, Bn, R_next, R_next)
    out, res = torch.zeros(n, dtype=torch.float16, device="cuda"), dev(sb.uniform_half(4, n))
    with operand_swap(swap):
        op = sb.SpconvChainOp().initialize(f, Bn, H, H, stride, x, out, R_next, R_next, alpha=0.25, relu=True)
        if residual:
            op.set_residual(res, None)
    op(torch.cuda.current_stream())
    torch.cuda.synchronize()
    f.device_status()
    return host(out).view(np.uint16).copy(), op._state


@pytest.mark.parametrize("V,Bn,H,Cc,R,stride,R_next,cols,variant,gather", [
    (64, 64, 14, 128, 3, 1, 1, 230, 0, 1),      # deep: tokens in lanes all the same
    (64, 8, 15, 128, 3, 1, 1, 230, 0, 1),       # ... of padded rows
    (64, 8, 15, 128, 3, 1, 3, 230, 1, 1),       # ... into a halo: rows
    (64, 8, 5, 128, 3, 1, 1, 230, 1, 1),        # a handful of items: rows
    (64, 64, 14, 256, 3, 1, 1, 1300, 1, 1),     # the MMAs bound it: rows
    (128, 64, 14, 256, 3, 1, 1, 1300, 0, 1),
    (128, 64, 14, 128, 1, 1, 3, 20, 0, 1),
    (128, 64, 14, 128, 1, 1, 1, 100, 0, 0),     # a stage and a half
    (128, 64, 14, 256, 1, 1, 1, 150, 0, 1),
    (128, 24, 13, 128, 3, 1, 1, 150, 0, 0),     # padded rows
    (128, 8, 7, 256, 1, 1, 1, 20, 0, 1),        # fewer items than SMs, 128-token tiles
    (128, 64, 14, 64, 3, 2, 1, 230, 0, 1),      # strided, a box per pixel
])
@pytest.mark.parametrize("residual", [False, True])
def test_chained_layers(V, Bn, H, Cc, R, stride, R_next, cols, variant, gather, residual, monkeypatch):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the item counts are of 148 SMs")
    F = V * (4 if Bn * H < 60 else 10)
    f = sb.BlockwiseSpFilter().init_random(F, R, R, Cc, V, 1, (cols + 0.5) / (R * R * Cc), True, 5, values="uniform")
    f.transform_and_sync_device()
    got, st = _chained(f, Bn, H, R, stride, R_next, residual, None, None, monkeypatch)
    assert (st.variant, st.gather) == (variant, gather)
    for swap in (0, 1):
        other, st = _chained(f, Bn, H, R, stride, R_next, residual, swap, 0, monkeypatch)
        assert (st.variant, st.gather) == (swap, 0)
        assert np.array_equal(got, other)
    assert np.abs(got.view(np.float16).astype(np.float32)).max() > 0


@pytest.mark.parametrize("V,Bn,H,Cc,F,R,stride,cols,permute,variant,rows,wide", [
    (64, 16, 14, 128, 1024, 3, 1, 230, True, 1, 0, 0),     # planes, tokens in lanes
    (64, 16, 14, 256, 1024, 3, 1, 1300, True, 1, 1, 0),    # ... filters in lanes
    (64, 31, 24, 64, 512, 1, 1, 20, True, 1, 0, 1),        # ... sixteen epilogue warps, a padding image
    (64, 31, 24, 64, 512, 1, 1, 40, True, 1, 0, 1),
    (128, 16, 14, 128, 2048, 3, 1, 100, True, 1, 0, 0),
    (64, 8, 28, 64, 512, 3, 1, 40, True, 0, 0, 0),         # less than a stage of columns, padded rows: positions
    (64, 9, 28, 64, 512, 1, 1, 40, True, 0, 0, 0),         # nine images in sixteen
    (64, 8, 14, 128, 512, 3, 1, 230, True, 0, 0, 0),       # fewer items than SMs
    (64, 16, 14, 128, 1024, 3, 1, 230, False, 0, 0, 0),    # nothing to permute
    (128, 16, 28, 256, 2048, 3, 2, 230, True, 1, 0, 0),
])
def test_nhwc_calls(V, Bn, H, Cc, F, R, stride, cols, permute, variant, rows, wide, monkeypatch):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the item counts are of 148 SMs")
    f = sb.BlockwiseSpFilter().init_random(F, R, R, Cc, V, 1, (cols + 0.5) / (R * R * Cc), permute, 5, values="uniform")
    f.transform_and_sync_device()
    x = dev(sb.uniform_half(3, Bn * H * H * Cc).reshape(Bn, H, H, Cc))
    bias = dev(sb.uniform_half(4, F))
    Ho = -(-H // stride)
    got = {}
    for planes in (None, "0", "1"):
        if planes:
            monkeypatch.setenv("SHFLBW_CONV_PLANES", planes)
        y = torch.full((Bn, Ho, Ho, F), float("nan"), dtype=torch.float16, device="cuda")
        op = sb.SpconvBlockwiseOp().initialize(f, Bn, H, H, stride, x, y, 0.25)
        st = op._state
        if planes:
            assert st.variant == int(planes)
        else:
            assert (st.variant, st.rows, st.wide) == (variant, rows, wide)
        out = []
        for b in (None, bias):
            op.run_with_bias(b, torch.cuda.current_stream())
            torch.cuda.synchronize()
            f.device_status()
            out.append(host(y).view(np.uint16).copy())
        got[planes] = out
    for planes in ("0", "1"):
        assert all(np.array_equal(a, b) for a, b in zip(got[None], got[planes]))
    assert not np.array_equal(*got[None])


def test_planes_that_do_not_fit_the_fixed_scratch_give_way_to_positions():
    """Seven images, whose planes hold eight: at the smallest image whose planes are beyond the array the positions fit."""
    H, Bn = 40, 7
    f = sb.BlockwiseSpFilter().init_random(192, 1, 1, 8, 64, 1, 0.5, True, 9, values="uniform")
    f.transform_and_sync_device()
    need = lambda images: 2 * 8 * H * H * 8 + 2 * images * H * H * f.F
    while need(8) <= _cabi.STATIC_SCRATCH_BYTES:
        H += 1
    assert need(7) + 512 <= _cabi.STATIC_SCRATCH_BYTES < need(8)
    x = dev(sb.uniform_half(3, Bn * H * H * 8).reshape(Bn, H, H, 8))
    y, want = (torch.full((Bn, H, H, f.F), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2))
    s = torch.cuda.current_stream()
    rc = _cabi.lib().shflbw_spconv_exec_static_scratch(f._h, Bn, H, H, 1, x.data_ptr(), y.data_ptr(), 1.0, s.cuda_stream)
    assert rc == 0
    op = sb.SpconvBlockwiseOp().initialize(f, Bn, H, H, 1, x, want)
    assert op._state.variant == 1
    op(s)
    torch.cuda.synchronize()
    f.device_status()
    assert torch.equal(y.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("V,blocks,K,N,cols,beta,variant", [
    (64, 40, 512, 4096, 40, 0.0, 2), (64, 40, 512, 4096, 100, 0.0, 1), (64, 40, 512, 1024, 40, 0.0, 1),    # whole sectors
    (64, 40, 512, 4104, 90, 0.0, 2), (64, 40, 512, 4104, 130, 0.0, 0), (64, 40, 512, 1032, 40, 0.0, 0),    # not
    (64, 10, 512, 504, 130, 0.0, 1), (64, 10, 512, 504, 40, 0.0, 0), (64, 10, 512, 40, 20, 0.0, 1),
    (64, 40, 512, 4096, 120, -1.5, 2), (64, 40, 512, 4096, 300, -1.5, 0), (64, 4, 2048, 512, 1700, -1.5, 1), (64, 4, 2048, 24, 300, -1.5, 1),
    (128, 20, 512, 4096, 20, 0.0, 1), (128, 20, 512, 4104, 300, 0.0, 0), (128, 20, 512, 64, 100, 0.0, 1), (128, 20, 512, 4096, 300, -1.5, 0),
    (128, 2, 512, 8, 300, -1.5, 1),
])
def test_spmm(V, blocks, K, N, cols, beta, variant):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the item counts are of 148 SMs")
    m = sb.BlockwiseSpMatrix().init_random(V * blocks, K, V, 1, (cols + 0.5) / K, True, 5, values="uniform")
    B = sb.uniform_half(6, K * N).reshape(K, N)
    Cm = sb.uniform_half(7, m.nrow * N).reshape(m.nrow, N) if beta else None
    D, op = run_spmm(m, N, B, alpha=0.5, Cm=Cm, beta=beta)
    assert op._state.variant == variant
    for swap in (0, 1):
        with operand_swap(swap):
            E, op = run_spmm(m, N, B, alpha=0.5, Cm=Cm, beta=beta)
        assert (op._state.variant == 1) == bool(swap)
        assert np.array_equal(D.view(np.uint16), E.view(np.uint16))
    assert np.abs(D.astype(np.float32)).max() > 0


def test_rows_that_start_between_sectors_keep_tokens_in_lanes():
    m = sb.BlockwiseSpMatrix().init_random(64 * 40, 512, 64, 1, 0.2, True, 5, values="uniform")
    m.transform_and_sync_device()
    B = dev(sb.uniform_half(6, 512 * 4096).reshape(512, 4096))
    flat = torch.zeros(m.nrow * 4096 + 8, dtype=torch.float16, device="cuda")
    s = torch.cuda.current_stream()
    got = []
    for off, variant in ((0, 1), (8, 0)):
        D = flat[off:off + m.nrow * 4096]
        op = sb.SpmmBlockwiseOp().initialize(m, 4096, B, D)
        assert op._state.variant == variant
        op(s)
        torch.cuda.synchronize()
        m.device_status()
        got.append(host(D).view(np.uint16).copy())
    assert np.array_equal(*got)


@pytest.mark.parametrize("V,M,K,N,density,tile", (
    (128, 2944, 1504, 1752, 0.164, 128), (64, 9536, 1256, 232, 0.093, 128), (32, 5504, 2744, 152, 0.181, 128), (16, 400, 2312, 1872, 0.095, 128),
    (32, 832, 400, 1520, 0.099, 256), (16, 976, 2488, 1184, 0.226, 128), (64, 896, 520, 5536, 0.35, 256), (16, 3072, 768, 1000, 0.25, 128), (16, 3072, 768, 1024, 0.25, 256)))
def test_spmm_tile_by_rounds(monkeypatch, V, M, K, N, density, tile):
    """Two rounds of 256-token items or three of 128: the rule's sides, and the same bits either way."""
    m = sb.BlockwiseSpMatrix().init_random(M, K, V, 1, density, True, 7, values="uniform")
    m.transform_and_sync_device()
    b = (torch.rand(K, N, device="cuda") * 2 - 1).half()
    got = []
    for forced in (None, "256", "128"):
        if forced: monkeypatch.setenv("SHFLBW_TILE", forced)
        d = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        op = sb.SpmmBlockwiseOp().initialize(m, N, b, d)
        if not forced and torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert op._state.tokens_per_cta == tile
        op()
        torch.cuda.synchronize()
        got.append(d)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("K,N,M,cols,beta,tile", (
    (2816, 2392, 3728, 180, 1.0, 256), (2816, 2392, 3728, 180, 0.0, 256), (3200, 1400, 4096, 180, 1.0, 256),      # many rounds
    (768, 1000, 3072, 180, 1.0, 128), (1776, 1288, 1856, 300, 1.0, 128), (1360, 2696, 1360, 180, 0.0, 256)))
def test_tiles_of_16_rows_and_ragged_columns(monkeypatch, K, N, M, cols, beta, tile):
    """Rows of B between sectors: 128-token items where the rounds that they save pay for their epilogues, C among them."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rounds are of 148 SMs")
    m = sb.BlockwiseSpMatrix().init_random(M, K, 16, 1, (cols + 0.5) / K, True, 7, values="uniform")
    m.transform_and_sync_device()
    b, c = ((torch.rand(r, N, device="cuda") * 2 - 1).half() for r in (K, M))
    got = []
    for forced in (None, "256", "128"):
        if forced: monkeypatch.setenv("SHFLBW_TILE", forced)
        d = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        op = sb.SpmmBlockwiseOp().initialize(m, N, b, 1.0, c, beta, d) if beta else sb.SpmmBlockwiseOp().initialize(m, N, b, d)
        assert forced or op._state.tokens_per_cta == tile
        op()
        torch.cuda.synchronize()
        got.append(d)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("V,B,H,W,C,F,R,stride,cols,variant", (
    (64, 3, 39, 11, 616, 3712, 1, 2, 197, 1), (128, 9, 5, 5, 64, 3840, 3, 1, 303, 1), (64, 18, 7, 7, 632, 3072, 3, 2, 267, 1),   # many filters:
    (128, 27, 13, 13, 888, 2432, 1, 2, 356, 1), (64, 6, 9, 9, 176, 1088, 3, 1, 300, 1),                    # planes whatever the batch and the tile
    (64, 3, 9, 9, 176, 1088, 3, 1, 300, 0), (64, 6, 9, 9, 176, 1024, 3, 1, 300, 0),                        # eight planes for three images; fewer filters
    (64, 46, 46, 46, 328, 2112, 1, 2, 135, 0), (128, 58, 15, 8, 584, 3840, 1, 1, 40, 1), (64, 48, 58, 58, 64, 640, 1, 1, 40, 1)))   # beyond the L2; not; few filters
def test_planes_by_filters_and_bytes(V, B, H, W, C, F, R, stride, cols, variant, monkeypatch):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the item counts are of 148 SMs")
    f = sb.BlockwiseSpFilter().init_random(F, R, R, C, V, 1, (cols + 0.5) / (R * R * C), True, 5, values="uniform")
    f.transform_and_sync_device()
    x = (torch.rand(B, H, W, C, device="cuda") * 2 - 1).half()
    got = []
    for planes in (None, "0", "1"):
        if planes:
            monkeypatch.setenv("SHFLBW_CONV_PLANES", planes)
        y = torch.full((B, -(-H // stride), -(-W // stride), F), float("nan"), dtype=torch.float16, device="cuda")
        op = sb.SpconvBlockwiseOp().initialize(f, B, H, W, stride, x, y, 0.25)
        assert op._state.variant == (int(planes) if planes else variant)
        op(torch.cuda.current_stream())
        torch.cuda.synchronize()
        got.append(y)
    f.device_status()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
