"""States are PODs with public addresses: a caller may bind one once and exchange its buffers between calls."""
import numpy as np
import pytest
import torch

import oracle_api as oa
import shflbw_sparse_nn_b200 as sb
from shflbw_sparse_nn_b200 import blockwise as bw
from conftest import assert_close_fp16
from gpu_util import dev, epilogue_warps, host, operand_swap, run_spconv, run_spmm, tile

pytestmark = pytest.mark.gpu


def _call(op, m):
    op(torch.cuda.current_stream())
    torch.cuda.synchronize()
    m.device_status()


@pytest.mark.parametrize("V,swap", [(16, 0), (32, 0), (64, 0), (64, 1), (128, 0), (128, 1)])
def test_spmm_state_follows_exchanged_operands(V, swap):
    """B exchanged, and B and D exchanged for narrower ones: the same bits as a state made for those buffers."""
    M, K, N = 2 * V, 256, 264
    m = sb.BlockwiseSpMatrix().init_random(M, K, V, 1, 0.3, True, 5 + V, values="uniform")
    B0, B1 = (sb.uniform_half(6 + i, K * N).reshape(K, N) for i in range(2))
    narrow = np.ascontiguousarray(B1[:, :N - 8])
    with operand_swap(swap):
        D0, op = run_spmm(m, N, B0)
        D1, _ = run_spmm(m, N, B1)
        D2, _ = run_spmm(m, N - 8, narrow)
    b1, bn = dev(B1), dev(narrow)
    d = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    dn = torch.full((M, N - 8), float("nan"), dtype=torch.float16, device="cuda")
    first = (op._state.B, op._state.D)
    op._state.B, op._state.D = b1.data_ptr(), d.data_ptr()
    _call(op, m)
    assert np.array_equal(host(d).view(np.uint16), D1.view(np.uint16))
    op._state.B, op._state.D, op._state.N = bn.data_ptr(), dn.data_ptr(), N - 8
    _call(op, m)
    assert np.array_equal(host(dn).view(np.uint16), D2.view(np.uint16))
    op._state.N = N
    op._state.B, op._state.D = first[0], d.data_ptr()
    _call(op, m)
    assert np.array_equal(host(d).view(np.uint16), D0.view(np.uint16))


@pytest.mark.parametrize("V,R", [(32, 3), (64, 3), (64, 1)])
def test_spconv_state_follows_exchanged_operands(V, R):
    B, H, W, C = 8, 7, 8, 16
    f = sb.BlockwiseSpFilter().init_random(2 * V, R, R, C, V, 1, 0.4, True, 9 + V, values="uniform")
    x0, x1 = (sb.uniform_half(10 + i, B * H * W * C).reshape(B, H, W, C) for i in range(2))
    _, op = run_spconv(f, B, H, W, 1, x0)
    y1, _ = run_spconv(f, B, H, W, 1, x1)
    xd = dev(x1)
    yd = torch.full((B, H, W, 2 * V), float("nan"), dtype=torch.float16, device="cuda")
    op._state.ifmap, op._state.ofmap = xd.data_ptr(), yd.data_ptr()
    _call(op, f)
    assert np.array_equal(host(yd).view(np.uint16), y1.view(np.uint16))


@pytest.mark.parametrize("Bn,H,W,R,stride,V,gather,row_pix", [
    (8, 9, 16, 3, 1, 64, 1, 16),      # rows of whole 64-token boxes
    (3, 9, 13, 3, 1, 32, 1, 16),      # rounded up to them
    (64, 9, 13, 3, 2, 64, 1, 7),      # strided, a box per pixel
    (16, 9, 9, 3, 2, 64, 0, 5),       # strided, no whole box: cp.async
    (5, 9, 13, 1, 1, 128, 1, 13),     # no halo
])
def test_spconv_state_says_how_it_gathers(Bn, H, W, R, stride, V, gather, row_pix, monkeypatch):
    """The gather and the pixels of a row are the plan's, and its item count is theirs; the other gather by request."""
    f = sb.BlockwiseSpFilter().init_random(2 * V, R, R, 16, V, 1, 0.4, True, 19, values="uniform")
    x = sb.uniform_half(20, Bn * H * W * 16).reshape(Bn, H, W, 16)
    for env, want_gather, want_pix in ((None, gather, row_pix), ("0", 0, -(-W // stride))):
        if env is None:
            monkeypatch.delenv("SHFLBW_GATHER", raising=False)
        else:
            monkeypatch.setenv("SHFLBW_GATHER", env)
        _, op = run_spconv(f, Bn, H, W, stride, x)
        st = op._state
        assert (st.gather, st.row_pix) == (want_gather, want_pix)
        assert st.num_items == 2 * -(-(st.Ho * st.row_pix * st.Bp) // st.tokens_per_cta)


@pytest.mark.parametrize("density,residual,tokens,gather,variant", [
    (0.05, False, 128, 1, 0), (0.05, True, 128, 1, 0), (0.05, False, 256, 0, 0), (0.6, False, 128, 0, 0), (0.6, True, 256, 0, 0), (0.9, True, 256, 1, 1),
])
def test_chained_layers_of_128_rows_gather_by_what_is_faster_for_them(density, residual, tokens, gather, variant):
    """Tokens in lanes: TMA for one stage of columns in 128-token tiles, else cp.async; rows in lanes: TMA.  Against the
    oracle either way, max(1e-2 * |ref|, 1e-3) as for every fp16 result of fp32 sums, with a residual's fp16 sum on top."""
    Bn, H, W, C, V, F = 8, 6, 9, 240, 128, 256
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, C, V, 1, density, True, 23, values="uniform")
    f.transform_and_sync_device()
    x = sb.uniform_half(24, Bn * H * W * C).reshape(Bn, H, W, C)
    s = torch.cuda.current_stream()
    b0 = torch.zeros(sb.chain_buffer_elems(C, H, W, Bn), dtype=torch.float16, device="cuda")
    b1 = torch.zeros(sb.chain_buffer_elems(F, H, W, Bn), dtype=torch.float16, device="cuda")
    r = dev(sb.uniform_half(25, Bn * H * W * F).reshape(Bn, H, W, F))
    br = torch.zeros_like(b1)
    y = torch.empty((Bn, H, W, F), dtype=torch.float16, device="cuda")
    sb.chain_import_nhwc(dev(x), Bn, H, W, C, 1, 1, b0, s)
    sb.chain_import_nhwc(r, Bn, H, W, F, 1, 1, br, s)
    with tile(tokens):
        op = sb.SpconvChainOp().initialize(f, Bn, H, W, 1, b0, b1)
    if residual:
        op.set_residual(br, None)
    op(s)
    sb.chain_export_nhwc(b1, Bn, H, W, F, 1, 1, f, y, s)
    torch.cuda.synchronize()
    f.device_status()
    assert (op._state.variant, op._state.gather) == (variant, gather)
    want = np.asarray(oa.spconv_ref_nhwc(Bn, H, W, C, F, 1, 1, 1, V, f.indptr, f.indices, f.values, f.row_permute_ids, x), np.float32)
    if residual:
        want = want.reshape(Bn, H, W, F) + host(r).astype(np.float32)
    assert_close_fp16(host(y), want.reshape(Bn, H, W, F), what=f"density {density}")


@pytest.mark.parametrize("H,Bn,V,F,density,gather,tokens", [
    (17, 24, 64, 128, 0.9, 0, 128),     # 55 tiles of 128 tokens, two blocks; rows of 24 pixels would make two rounds of 128
    (17, 24, 64, 128, 0.2, 1, 256),     # less than a stage of columns a block: one round of 256 all the same
    (17, 24, 128, 256, 0.2, 0, 128),    # ... not at 128 rows
    (17, 24, 32, 64, 0.9, 0, 128),
    (17, 24, 64, 1024, 0.6, 0, 256),    # four rounds of items; five with the rows padded
    (17, 24, 32, 512, 0.6, 0, 256),     # ... of 1.41 times the tokens
    (19, 24, 32, 512, 0.6, 1, 256),     # ... of 1.26 times
    (18, 15, 64, 1728, 0.06, 1, 256),   # four rounds, five padded, of less than half a stage
    (10, 6, 128, 1792, 0.06, 0, 128),   # one round either way, but 140 items for 98
])
def test_padded_rows_are_weighed_in_the_tiles_that_each_side_takes(H, Bn, V, F, density, gather, tokens):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the item counts are of 148 SMs")
    C = 16
    f = sb.BlockwiseSpFilter().init_random(F, 3, 3, C, V, 1, density, True, 27, values="uniform")
    x = sb.uniform_half(28, Bn * H * H * C).reshape(Bn, H, H, C)
    y, op = run_spconv(f, Bn, H, H, 1, x)
    st = op._state
    whole = {17: 24, 19: 24, 18: 20}.get(H)                      # pixels of a row in whole boxes
    assert (st.gather, st.tokens_per_cta, st.row_pix) == (gather, tokens, whole if gather else H)
    n = 2 * H * H                                                # two images suffice for the oracle
    want = oa.spconv_ref_nhwc(2, H, H, C, F, 3, 3, 1, V, f.indptr, f.indices, f.values, f.row_permute_ids, x[:2])
    assert_close_fp16(y[:2].reshape(n, F), np.asarray(want).reshape(n, F), what=f"V={V} F={F}")


@pytest.mark.parametrize("V,K,N,dense,gather", [
    (16, 256, 8, False, 0), (32, 1024, 8, False, 0), (64, 1024, 8, False, 0), (128, 256, 8, False, 0), (16, 256, 24, True, 0),
    (32, 1032, 8, False, 1), (32, 1544, 8, True, 0), (16, 3080, 8, True, 1), (16, 512, 16, True, 1), (16, 256, 40, True, 1),
])
@pytest.mark.parametrize("beta", [0.0, -1.5])
def test_spmm_on_few_shared_lines_gathers_by_cp_async(V, K, N, dense, gather, beta, monkeypatch):
    """Rows that share sectors, wanted by many blocks: the same bits as by TMA, and the oracle's values; a linear layer's too."""
    counts = ([K, K, K // 2 + 1, K, 17, 0] if dense else [0, 1, K // 4, K // 2, K - 1, 17]) * (56 if N == 24 else 28)
    M = V * len(counts)
    rng = np.random.default_rng(K + V)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    indices = np.concatenate([np.sort(rng.choice(K, c, replace=False)) for c in counts]).astype(np.int32)
    m = sb.BlockwiseSpMatrix.from_arrays(M, K, V, indptr, indices, sb.uniform_half(3, indices.size * V),
                                         rng.permutation(M).astype(np.int32))
    B = sb.uniform_half(30, K * N).reshape(K, N)
    Cm = sb.uniform_half(31, M * N).reshape(M, N) if beta else None
    monkeypatch.delenv("SHFLBW_GATHER", raising=False)
    D, op = run_spmm(m, N, B, alpha=0.5, Cm=Cm, beta=beta)
    bias, bd = dev(sb.uniform_half(32, M)), dev(B)
    out, forced = (torch.empty((M, N), dtype=torch.float16, device="cuda") for _ in range(2))
    bw.linear_exec(m, N, None, bias, bd, N, out, torch.cuda.current_stream())
    monkeypatch.setenv("SHFLBW_GATHER", "1")
    E, op_tma = run_spmm(m, N, B, alpha=0.5, Cm=Cm, beta=beta)
    bw.linear_exec(m, N, None, bias, bd, N, forced, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert (op._state.gather, op_tma._state.gather) == (gather, 1)
    assert np.array_equal(D.view(np.uint16), E.view(np.uint16))
    assert torch.equal(out.view(torch.int16), forced.view(torch.int16))
    if K <= 256:                                                 # (a quick oracle)
        want = oa.spmm_ref(M, N, V, indptr, indices, m.values, m.row_permute_ids, B, 0.5, Cm, beta)
        assert_close_fp16(D, np.asarray(want).reshape(M, N), what=f"V={V} K={K} N={N}")


@pytest.mark.parametrize("V,swap,ew,tokens", [(16, 0, 8, 256), (32, 0, 8, 128), (64, 0, 8, 256), (64, 1, 8, 256), (64, 0, 16, 256), (128, 1, 8, 256)])
def test_linear_layers_where_cp_async_is_asked_for(V, swap, ew, tokens, monkeypatch):
    """With a bias, and with sixteen epilogue warps, the SpMM kernels of 256-token tiles gather by TMA only: asking for
    the other gather changes neither the bits nor what is accepted."""
    K, N, M = 192, 200, 4 * V
    m = sb.BlockwiseSpMatrix().init_random(M, K, V, 1, 0.3, True, 33 + V, values="uniform")
    m.transform_and_sync_device()
    B, bias = sb.uniform_half(34, K * N).reshape(K, N), sb.uniform_half(35, M)
    bd, biasd, got = dev(B), dev(bias), []
    for env in ("1", "0"):
        monkeypatch.setenv("SHFLBW_GATHER", env)
        out, plain = (torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2))
        with operand_swap(swap), epilogue_warps(ew), tile(tokens):
            bw.linear_exec(m, N, None, biasd, bd, N, out, torch.cuda.current_stream())
            op = sb.SpmmBlockwiseOp().initialize(m, N, bd, plain)
        _call(op, m)
        assert op._state.gather == (1 if env == "1" or ew == 16 else 0)
        got.append((host(out), host(plain)))
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.uint16), b.view(np.uint16))
    perm = m.row_permute_ids
    want = np.asarray(oa.spmm_ref(M, N, V, m.indptr, m.indices, m.values, perm, B)).reshape(M, N) + bias.astype(np.float32)[:, None]
    assert_close_fp16(got[1][0], want, what=f"V={V}")
