"""The TMA gather against the cp.async gather (SHFLBW_GATHER=0) and the CPU oracle.  Both feed the same
MMAs in the same order, so their outputs are equal bit for bit; the oracle is met at the usual tolerance of
an fp16 result with fp32 sums, max(1e-2 * |ref|, 1e-3)."""
import numpy as np
import pytest
import torch

import oracle_api as oa
import shflbw_sparse_nn_b200 as sb
from conftest import assert_close_fp16
from gpu_util import dev, epilogue_warps, host, operand_swap, run_spconv, run_spmm, tile

pytestmark = pytest.mark.gpu


def _both(monkeypatch, call):
    """(TMA, cp.async) results of call()."""
    monkeypatch.delenv("SHFLBW_GATHER", raising=False)
    got = call()
    monkeypatch.setenv("SHFLBW_GATHER", "0")
    return got, call()


@pytest.mark.parametrize("V,swap", [(16, 0), (32, 0), (64, 0), (64, 1), (128, 0), (128, 1)])
@pytest.mark.parametrize("tokens,N", [(128, 8), (128, 136), (256, 72), (256, 1000)])
def test_spmm(V, swap, tokens, N, monkeypatch):
    """Every block height in both orientations, boxes of 64 tokens that N fills, cuts and never reaches; row
    blocks that end before, at and after a quad's, a warp's half and a whole stage of 64 columns, empty ones first,
    between and last; more stages than the ring."""
    counts = [0, 1, 16, 17, 32, 33, 64, 65, 0, 128, 400, 0]
    K, M = 448, V * len(counts)
    rng = np.random.default_rng(V + N)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    indices = np.concatenate([np.sort(rng.choice(K, c, replace=False)) for c in counts]).astype(np.int32)
    m = sb.BlockwiseSpMatrix.from_arrays(M, K, V, indptr, indices, sb.uniform_half(3, indices.size * V),
                                         rng.permutation(M).astype(np.int32))
    B = sb.uniform_half(4, K * N).reshape(K, N)
    B[5, N // 2], B[6, 0], B[7, N - 1] = np.inf, -np.inf, np.nan      # stay in their own column
    Cm = sb.uniform_half(5, M * N).reshape(M, N)
    with operand_swap(swap):
        (D, op), (E, op_cp) = _both(monkeypatch, lambda: run_spmm(m, N, B, alpha=0.5, Cm=Cm, beta=-1.5, tokens=tokens))
    assert (op._state.gather, op_cp._state.gather, op._state.variant) == (1, 0, swap)
    assert np.array_equal(D.view(np.uint16), E.view(np.uint16))
    ok = np.ones(N, bool)
    ok[[0, N // 2, N - 1]] = False
    want = oa.spmm_ref(M, N, V, indptr, indices, m.values, m.row_permute_ids, B, 0.5, Cm, -1.5)
    assert_close_fp16(D[:, ok], np.asarray(want).reshape(M, N)[:, ok], what=f"V={V} swap={swap} N={N}")


@pytest.mark.parametrize("Bn,H,W,Cc,R,stride,V,tma", [
    (64, 6, 5, 16, 3, 1, 64, True),       # a box is one pixel
    (64, 9, 7, 16, 3, 2, 64, True),       # and so may be strided
    (128, 5, 5, 16, 3, 2, 32, True),
    (8, 9, 16, 24, 3, 1, 128, True),      # rows of whole boxes
    (3, 9, 13, 24, 3, 1, 64, True),       # rows padded to whole boxes
    (16, 14, 14, 24, 3, 1, 32, True),
    (24, 7, 20, 16, 3, 1, 16, True),      # three boxes to eight pixels
    (5, 11, 9, 40, 1, 1, 32, True),       # no halo: boxes run through pixels and rows
    (5, 13, 13, 40, 1, 2, 64, True),      # strided 1x1, staged compactly
    (1, 7, 1, 64, 1, 1, 64, True),        # fewer tokens than a box
    (16, 9, 9, 16, 3, 2, 64, False),      # strided taps of less than a box
])
@pytest.mark.parametrize("permute", [True, False])
def test_spconv(Bn, H, W, Cc, R, stride, V, tma, permute, monkeypatch):
    F = 2 * V
    f = sb.BlockwiseSpFilter().init_random(F, R, R, Cc, V, 1, 0.5, permute, 41 + V, values="uniform")
    x = sb.uniform_half(42, Bn * H * W * Cc).reshape(Bn, H, W, Cc)
    (y, op), (y_cp, op_cp) = _both(monkeypatch, lambda: run_spconv(f, Bn, H, W, stride, x))
    assert (op._state.gather, op_cp._state.gather) == (int(tma), 0)
    assert np.array_equal(y.view(np.uint16), y_cp.view(np.uint16))
    want = oa.spconv_ref_nhwc(Bn, H, W, Cc, F, R, R, stride, V, f.indptr, f.indices, f.values,
                              f.row_permute_ids if permute else None, x)
    assert_close_fp16(y, want, what="TMA gather")


def test_padding_that_costs_a_round_of_items_keeps_the_other_gather():
    """14 pixels of 16 images count as 16 in boxes of 64 tokens: where that makes three rounds of items four, the
    plan stays with cp.async."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = 3 * sms // 13                                       # 13 tiles of 256 tokens each; 14 with the rows padded
    f = sb.BlockwiseSpFilter().init_random(blocks * 64, 3, 3, 16, 64, 1, 0.1, True, 7, values="uniform")
    x = sb.uniform_half(8, 16 * 14 * 14 * 16).reshape(16, 14, 14, 16)
    y, op = run_spconv(f, 16, 14, 14, 1, x)
    padded = -(-14 * blocks // sms)
    assert op._state.num_items == (13 if padded > 3 else 14) * blocks
    want = oa.spconv_ref_nhwc(16, 14, 14, 16, blocks * 64, 3, 3, 1, 64, f.indptr, f.indices, f.values, f.row_permute_ids, x)
    assert_close_fp16(y, want, what="the other gather")


@pytest.mark.parametrize("Bn,H,stride,V,swap,ew", [(8, 9, 1, 64, 1, None), (8, 9, 1, 64, 0, 8), (8, 9, 1, 64, 0, 16),
                                                   (64, 7, 2, 64, 0, 16), (3, 13, 1, 128, 1, None), (64, 6, 2, 32, 0, None)])
@pytest.mark.parametrize("residual", [True, False])
def test_chained_layer(Bn, H, stride, V, swap, ew, residual, monkeypatch):
    """A 3x3 layer into the halo of another one, with ReLU and a residual."""
    W, Cc, F = H - 1, 16, 2 * V
    Ho, Wo = -(-H // stride), -(-W // stride)
    f = sb.BlockwiseSpFilter().init_random(F, 3, 3, Cc, V, 1, 0.4, True, 51, values="uniform")
    f.transform_and_sync_device()
    x = sb.uniform_half(52, Bn * H * W * Cc).reshape(Bn, H, W, Cc)
    s = torch.cuda.current_stream()

    def run():
        b0 = torch.zeros(sb.chain_buffer_elems(Cc, H, W, Bn, 3, 3), dtype=torch.float16, device="cuda")
        b1 = torch.zeros(sb.chain_buffer_elems(F, Ho, Wo, Bn, 3, 3), dtype=torch.float16, device="cuda")
        res = dev(sb.uniform_half(53, b1.numel()))
        sb.chain_import_nhwc(dev(x), Bn, H, W, Cc, 3, 3, b0, s)
        with operand_swap(swap), epilogue_warps(ew), tile(256 if ew == 16 else None):
            op = sb.SpconvChainOp().initialize(f, Bn, H, W, stride, b0, b1, 3, 3, alpha=0.5, relu=True)
            if residual:
                op.set_residual(res, None)
        op(s)
        torch.cuda.synchronize()
        f.device_status()
        return host(b1), op

    (got, op), (want, op_cp) = _both(monkeypatch, run)
    assert (op._state.gather, op_cp._state.gather) == (1, 0) and op._state.variant == op_cp._state.variant
    if ew == 16:                                                 # three gather warps either way (57 columns a block)
        assert op._state.variant == 2 and (op._state.producer_warps, op_cp._state.producer_warps) == (3, 3)
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16))
    assert np.abs(got.astype(np.float32)).max() > 0


def _blocks(counts, K, V, seed):
    rng = np.random.default_rng(seed)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    indices = np.concatenate([np.sort(rng.choice(K, c, replace=False)) for c in counts]).astype(np.int32)
    M = V * len(counts)
    return sb.BlockwiseSpMatrix.from_arrays(M, K, V, indptr, indices, sb.uniform_half(seed, indices.size * V),
                                            rng.permutation(M).astype(np.int32))


@pytest.mark.parametrize("V,swap,tokens", [(16, 0, 128), (16, 0, 256), (32, 0, 128), (32, 0, 256), (64, 0, 256), (64, 1, 128),
                                           (64, 1, 256), (128, 0, 256), (128, 1, 128), (128, 1, 256)])
@pytest.mark.parametrize("mixed", [True, False])
def test_spmm_with_several_items_per_cta(V, swap, tokens, mixed, monkeypatch):
    """A CTA's stages run on from item to item: blocks of every length in turn, empty ones among them, and blocks of
    three whole stages and a quarter of one only, where a warp may have no row in every fourth stage; the last token
    tile is cut.  More than three items for every SM."""
    counts = [0, 1, 16, 17, 32, 33, 64, 65, 0, 128, 200, 0] if mixed else [208]
    tiles, N = (8, 1000) if tokens == 128 else (4, 1000)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = -(-(3 * sms + 5) // tiles)
    counts = (counts * blocks)[:blocks]
    m = _blocks(counts, 224, V, 71 + V)
    B = sb.uniform_half(72, 224 * N).reshape(224, N)
    with operand_swap(swap):
        (D, op), (E, op_cp) = _both(monkeypatch, lambda: run_spmm(m, N, B, tokens=tokens))
    st = op._state
    assert (st.gather, op_cp._state.gather, st.variant) == (1, 0, swap) and st.num_items > 3 * sms >= 3 * st.grid_x
    assert np.array_equal(D.view(np.uint16), E.view(np.uint16))
    want = oa.spmm_ref(m.nrow, N, V, m.indptr, m.indices, m.values, m.row_permute_ids, B)
    assert_close_fp16(D, np.asarray(want).reshape(D.shape), what=f"V={V} swap={swap}")


@pytest.mark.parametrize("beta", [0.0, -1.5])
def test_spmm_by_sixteen_epilogue_warps_with_several_items_per_cta(beta):
    """Stages of 32 columns, a gather warp each; against the eight-warp kernel, which sums in the same order."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = _blocks(([0, 1, 16, 17, 32, 33, 64, 65, 0, 100, 48, 0] * sms)[:-(-(3 * sms + 5) // 4)], 224, 64, 73)
    B = sb.uniform_half(74, 224 * 1000).reshape(224, 1000)
    Cm = sb.uniform_half(75, m.nrow * 1000).reshape(m.nrow, 1000) if beta else None
    got = []
    for ew in (16, 8):
        with operand_swap(0), epilogue_warps(ew):
            D, op = run_spmm(m, 1000, B, alpha=0.5, Cm=Cm, beta=beta, tokens=256)
        assert (op._state.variant, op._state.gather) == (2 if ew == 16 else 0, 1) and op._state.num_items > 3 * sms
        got.append(D)
    assert np.array_equal(got[0].view(np.uint16), got[1].view(np.uint16))


@pytest.mark.parametrize("V,blocks,C,density,variant", [(16, 120, 16, 0.3, 0), (32, 60, 16, 0.3, 0), (64, 60, 16, 0.3, 0), (64, 60, 32, 0.8, 1),
                                                        (128, 60, 32, 0.8, 1)])
def test_spconv_with_several_items_per_cta(V, blocks, C, density, variant, monkeypatch):
    """Rows of 15 pixels that count as 16: eight tiles of 256 tokens, the boxes of an item others than those of the next."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    f = sb.BlockwiseSpFilter().init_random(V * blocks, 3, 3, C, V, 1, density, True, 81 + V, values="uniform")
    x = sb.uniform_half(82, 8 * 15 * 15 * C).reshape(8, 15, 15, C)
    (y, op), (y_cp, op_cp) = _both(monkeypatch, lambda: run_spconv(f, 8, 15, 15, 1, x, tokens=256))
    st = op._state
    assert (st.gather, op_cp._state.gather, st.variant, st.row_pix) == (1, 0, variant, 16) and st.num_items >= 3 * sms
    assert np.array_equal(y.view(np.uint16), y_cp.view(np.uint16))
    want = oa.spconv_ref_nhwc(1, 15, 15, C, f.F, 3, 3, 1, V, f.indptr, f.indices, f.values, f.row_permute_ids, x[:1])
    assert_close_fp16(y[:1], want, what=f"V={V}")


@pytest.mark.parametrize("V,C,density,ew", [(32, 16, 0.3, None), (64, 16, 0.1, 16), (64, 16, 0.6, 16), (64, 16, 0.6, 8), (64, 32, 0.8, None),
                                            (128, 32, 0.8, None)])
@pytest.mark.parametrize("residual", [True, False])
def test_chained_layer_with_several_items_per_cta(V, C, density, ew, residual, monkeypatch):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    Bn, H, F = 8, 15, 60 * V
    f = sb.BlockwiseSpFilter().init_random(F, 3, 3, C, V, 1, density, True, 91 + V, values="uniform")
    f.transform_and_sync_device()
    x = sb.uniform_half(92, Bn * H * H * C).reshape(Bn, H, H, C)
    res = dev(sb.uniform_half(93, sb.chain_buffer_elems(F, H, H, Bn, 3, 3)))
    s = torch.cuda.current_stream()

    def run():
        b0 = torch.zeros(sb.chain_buffer_elems(C, H, H, Bn, 3, 3), dtype=torch.float16, device="cuda")
        b1 = torch.zeros(res.numel(), dtype=torch.float16, device="cuda")
        sb.chain_import_nhwc(dev(x), Bn, H, H, C, 3, 3, b0, s)
        with epilogue_warps(ew), tile(256):
            op = sb.SpconvChainOp().initialize(f, Bn, H, H, 1, b0, b1, 3, 3, alpha=0.5)
            if residual:
                op.set_residual(res, "same")
        op(s)
        y = torch.empty((Bn, H, H, F), dtype=torch.float16, device="cuda")
        sb.chain_export_nhwc(b1, Bn, H, H, F, 3, 3, f, y, s)
        torch.cuda.synchronize()
        f.device_status()
        return host(b1), host(y), op

    (got, y, op), (want, _, op_cp) = _both(monkeypatch, run)
    assert (op._state.gather, op_cp._state.gather) == (1, 0) and op._state.variant == op_cp._state.variant == (2 if ew == 16 else int(C == 32))
    assert op._state.num_items >= 3 * sms
    if ew == 16:                                                 # two gather warps beside a residual and few columns
        assert op._state.producer_warps == (2 if residual and density == 0.1 else 3) and op_cp._state.producer_warps == 3
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16))
    if not residual:
        ref = oa.spconv_ref_nhwc(1, H, H, C, F, 3, 3, 1, V, f.indptr, f.indices, f.values, f.row_permute_ids, x[:1], 0.5)
        assert_close_fp16(y[:1], ref, what=f"V={V}")
