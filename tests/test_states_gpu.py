"""States are PODs with public addresses: a caller may bind one once and exchange its buffers between calls."""
import numpy as np
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from gpu_util import dev, host, operand_swap, run_spconv, run_spmm

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
