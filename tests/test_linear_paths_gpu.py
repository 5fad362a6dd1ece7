"""ShflBWLinear: the transpose kernel and the bias added in the SpMM epilogue, against the plain
operator on a transposed copy and torch's fp16 add.  Both round the product to fp16 and then the
sum, so the results are the same bits."""
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from shflbw_sparse_nn_b200 import blockwise as bw
from gpu_util import epilogue_warps, operand_swap, tile
from shflbw_sparse_nn_b200.nn import ShflBWLinear

pytestmark = pytest.mark.gpu


def _plain(m, x2, bias):
    """[tokens][M] from SpmmBlockwiseOp on a padded transposed copy, bias added by torch."""
    n = -(-x2.shape[0] // 8) * 8
    xt = torch.zeros((m.ncol, n), dtype=torch.float16, device="cuda")
    xt[:, :x2.shape[0]] = x2.t()
    out = torch.empty((m.nrow, n), dtype=torch.float16, device="cuda")
    sb.SpmmBlockwiseOp().initialize(m, n, xt, out)(torch.cuda.current_stream())
    if bias is not None:
        out += bias[:, None]
    return out[:, :x2.shape[0]].t()


@pytest.mark.parametrize("V,K,tokens,swap,ew,t", [
    (64, 320, 1, None, None, None), (64, 320, 37, 1, None, 128), (64, 328, 65, 0, None, 128), (128, 320, 63, 1, None, 128),
    (32, 203, 8, None, None, None),                  # K % 8 != 0: 2-byte loads
    (64, 203, 300, 1, None, 256), (16, 77, 130, None, None, None),
    (64, 200, 256 * 40 + 5, 0, 16, 256),             # sixteen epilogue warps, ring of eight stages
    (64, 64, 256 * 40 + 5, 0, 16, 256),              # of six
    (64, 640, 256 * 40 + 13, 1, None, 256),          # TMA gather
    (64, 640, 256 * 40 + 3, 1, None, 256),           # and N % 16 == 8: 16-byte stores (32-byte ones above)
    (128, 320, 300, 1, None, 256), (128, 320, 120, 1, None, 128),
])
@pytest.mark.parametrize("bias", [True, False])
def test_forward_equals_operator_plus_bias_bit_for_bit(V, K, tokens, swap, ew, t, bias):
    m = sb.BlockwiseSpMatrix().init_random(512, K, V, 1, 0.3, True, 17, values="uniform")
    g = torch.Generator(device="cuda").manual_seed(tokens)
    b = (torch.rand(512, generator=g, device="cuda") * 2 - 1).half() if bias else None
    x = (torch.rand(tokens, K, generator=g, device="cuda") * 2 - 1).half()
    lin = ShflBWLinear(m, b).cuda()
    with operand_swap(swap), epilogue_warps(ew), tile(t):
        y = lin(x)
        want = _plain(m, x, b)
        xt = torch.zeros((K, -(-tokens // 8) * 8), dtype=torch.float16, device="cuda")
        xt[:, :tokens] = x.t()
        yt = lin.forward_feature_major(xt)
    torch.cuda.synchronize()
    m.device_status()
    assert y.shape == (tokens, 512) and torch.equal(y, want) and torch.equal(yt[:, :tokens].t(), want)


def test_inputs_that_are_not_contiguous_or_aligned():
    K, M = 256, 256
    m = sb.BlockwiseSpMatrix().init_random(M, K, 64, 1, 0.3, True, 18, values="uniform")
    lin = ShflBWLinear(m, torch.ones(M)).cuda()
    base = (torch.rand(41 * K + 3, device="cuda") * 2 - 1).half()
    x = base[3:].view(41, K)                              # 2-byte aligned only
    b = lin.bias
    assert torch.equal(lin(x), _plain(m, x, b))
    xs = (torch.rand(20, 2 * K, device="cuda") * 2 - 1).half()[:, ::2]      # strided
    assert torch.equal(lin(xs), _plain(m, xs, b))
    x3 = xs.reshape(4, 5, K)
    assert torch.equal(lin(x3), _plain(m, xs, b).reshape(4, 5, M))
    lin.bias = torch.rand(M, device="cuda")               # a bias that is not fp16 is added by torch
    assert torch.equal(lin(x), _plain(m, x, lin.bias))
    with pytest.raises(sb.ShflbwError):
        lin(x[:0])
    torch.cuda.synchronize()
    m.device_status()


@pytest.mark.parametrize("tokens", [512, 4099])
def test_input_in_the_operands_order_is_copied_once(tokens):
    """The result of one layer is feature-major memory: as the input of the next it needs no transposed copy."""
    M, K = 256, 1024
    m = sb.BlockwiseSpMatrix().init_random(M, K, 64, 1, 0.1, True, 19, values="uniform")
    lin = ShflBWLinear(m, None).cuda()
    padded = -(-tokens // 8) * 8
    x = (torch.rand(K, padded, device="cuda") * 2 - 1).half()[:, :tokens].t()
    lin(x)                                                # uploads the weights
    want = _plain(m, x, None)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    y = lin(x)
    peak = torch.cuda.max_memory_allocated() - before
    assert torch.equal(y, want) and peak <= (K + M) * padded * 2 + 4096        # the operand, the result, rounding
    m.device_status()


@pytest.mark.parametrize("direct", [0, 1])
@pytest.mark.parametrize("V,K,tokens,offset,swap,ew,t,gather", [
    (64, 320, 37, 0, 1, None, 128, None), (64, 328, 65, 0, 0, None, 128, None), (128, 320, 63, 0, 1, None, 128, None),
    (64, 640, 300, 0, 1, None, 256, "0"), (128, 320, 300, 0, 0, None, 256, None), (32, 320, 1, 0, None, None, None, None),
    (32, 203, 8, 0, None, None, None, None), (64, 203, 65, 0, 1, None, 256, None), (16, 77, 130, 0, None, None, None, None),   # K % 8 != 0: 2-byte loads,
    (64, 203, 300, 0, 0, None, 256, None), (128, 1031, 65, 0, None, None, None, None),                     # one and several 64-token tiles
    (64, 320, 65, 3, None, None, None, None), (32, 640, 130, 1, None, None, None, None), (16, 200, 300, 5, None, None, None, None),  # unaligned
    (64, 203, 256 * 40 + 5, 0, 0, 16, 256, None), (64, 64, 256 * 40 + 5, 1, 0, 16, 256, None),             # sixteen epilogue warps
])
def test_both_routes_equal_the_operator_bit_for_bit(monkeypatch, V, K, tokens, offset, swap, ew, t, gather, direct):
    """Few tokens go to the one-launch kernel by themselves: each case by it and by the transpose and the panel kernel."""
    monkeypatch.setenv("SHFLBW_LINEAR_DIRECT", str(direct))
    if gather is not None:
        monkeypatch.setenv("SHFLBW_GATHER", gather)
    m = sb.BlockwiseSpMatrix().init_random(512, K, V, 1, 0.3, True, 21, values="uniform")
    g = torch.Generator(device="cuda").manual_seed(tokens)
    b = (torch.rand(512, generator=g, device="cuda") * 2 - 1).half()
    buf = torch.full((tokens * K + 2 * K + offset,), float("nan"), dtype=torch.float16, device="cuda")
    x = buf[K + offset:][:tokens * K].view(tokens, K)        # amid NaN
    x.copy_(torch.rand(tokens, K, generator=g, device="cuda") * 2 - 1)
    lin = ShflBWLinear(m, b).cuda()
    with operand_swap(swap), epilogue_warps(ew), tile(t):
        y = lin(x)
        want = _plain(m, x, b)
    out = torch.empty((512, -(-tokens // 8) * 8), dtype=torch.float16, device="cuda")
    assert bw.linear_direct(m, tokens, x, b, out.shape[1], out, torch.cuda.current_stream()) == bool(direct)
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(y, want) and (not direct or torch.equal(out[:, :tokens].t(), want))
