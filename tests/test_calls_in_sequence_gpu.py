"""Calls on streams other than the default one, under capture, and of different kinds back to back.
Every kernel starts while the one before it still runs and waits for it on its own, so a missing wait
shows as a result that differs from the same calls with a synchronisation after each."""
import numpy as np
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from shflbw_sparse_nn_b200 import blockwise as bw
from gpu_util import dev
from shflbw_sparse_nn_b200.nn import ShflBWConv2d, ShflBWLinear

pytestmark = pytest.mark.gpu


def _modules():
    lin = ShflBWLinear(sb.BlockwiseSpMatrix().init_random(256, 128, 64, 1, 0.4, True, 1, values="uniform"),
                       dev(sb.uniform_half(2, 256))).cuda()
    conv = ShflBWConv2d(sb.BlockwiseSpFilter().init_random(96, 3, 3, 64, 32, 1, 0.2, False, 3, values="uniform"), 1,
                        dev(sb.uniform_half(4, 96))).cuda()
    x = dev(sb.uniform_half(5, 203 * 128).reshape(203, 128))
    xc = dev(sb.uniform_half(6, 5 * 9 * 9 * 64).reshape(5, 9, 9, 64)).permute(0, 3, 1, 2)
    return (lin, x), (conv, xc)


def test_modules_launch_on_the_current_stream():
    for module, x in _modules():
        want = module(x)
        late = torch.zeros_like(x)
        a = torch.rand(4096, 4096, device="cuda")
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(8):
                a = a @ a * 1e-4             # milliseconds during which `late` is still zero
            late.copy_(x)
            got = module(late)
        s.synchronize()
        assert torch.equal(got, want)


def test_modules_under_graph_capture():
    for module, x in _modules():
        static = x.clone()
        want = [module(x), module(-x)]
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = module(static)
        for value, w in ((x, want[0]), (-x, want[1])):
            static.copy_(value)
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, w)


@pytest.mark.parametrize("permute", [False, True])
def test_calls_of_different_kinds_back_to_back(permute):
    """Convolution -> SpMM -> chained layer -> convolution -> linear layer, each on the output of the one before."""
    n, h, c = 16, 16, 64                     # 4096 positions of 64 channels
    pos = n * h * h
    conv1 = sb.BlockwiseSpFilter().init_random(128, 3, 3, c, 32, 1, 0.2, permute, 11, values="uniform")
    mat = sb.BlockwiseSpMatrix().init_random(128, pos, 64, 1, 0.02, True, 12, values="uniform")    # K = positions
    layer = sb.BlockwiseSpFilter().init_random(64, 1, 1, 8, 32, 1, 0.9, True, 13, values="uniform")
    conv2 = sb.BlockwiseSpFilter().init_random(96, 1, 1, c, 32, 1, 0.4, permute, 14, values="uniform")
    for m in (conv1, mat, layer, conv2):
        m.transform_and_sync_device()
    lin = ShflBWLinear(sb.BlockwiseSpMatrix().init_random(256, 96, 64, 1, 0.5, True, 15, values="uniform"),
                       dev(sb.uniform_half(16, 256))).cuda()
    x = torch.zeros(n, h, h, c, dtype=torch.float16, device="cuda")
    y1 = torch.zeros(pos, 128, dtype=torch.float16, device="cuda")
    y2 = torch.zeros(128 * 128, dtype=torch.float16, device="cuda")          # read on as 8 planes of 2048
    y3 = torch.zeros(64 * 2048, dtype=torch.float16, device="cuda")          # read on as 8 images of 16 x 16 x 64
    y4 = torch.zeros(8 * 16 * 16, 96, dtype=torch.float16, device="cuda")
    ops = [sb.SpconvBlockwiseOp().initialize(conv1, n, h, h, 1, x, y1),
           sb.SpmmBlockwiseOp().initialize(mat, 128, y1, 0.125, None, 0.0, y2),
           sb.SpconvChainOp().initialize(layer, 8, 16, 16, 1, y2, y3, 1, 1, alpha=0.125),
           sb.SpconvBlockwiseOp().initialize(conv2, 8, 16, 16, 1, y3, y4, 0.125)]
    inputs = [dev(sb.uniform_half(20 + i, x.numel()).reshape(x.shape)) for i in range(8)]
    stream = torch.cuda.current_stream()

    def run(wait):
        out = []
        for value in inputs:
            x.copy_(value)
            for op in ops:
                wait()
                op(stream)
            wait()
            out.append(lin(y4))
            ops[0](stream)                   # and a call that nothing depends on
            wait()
        torch.cuda.synchronize()
        return out

    want = run(torch.cuda.synchronize)
    assert all(torch.isfinite(w).all() and w.abs().max() > 0 for w in want)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(lambda: None), want))
    for m in (conv1, mat, layer, conv2, lin.spmat):
        m.device_status()


def test_few_tokens_between_kernels_that_start_each_other_early():
    """SpMM -> one-launch linear layer -> SpMM on the same buffers every time: each reads what the kernel before has just written, and
    writes what the one behind it was still reading a call ago."""
    K, tokens = 4096, 64
    first = sb.BlockwiseSpMatrix().init_random(tokens, K, 64, 1, 0.5, True, 41, values="uniform")     # one block: 32 stages on one SM
    layer = sb.BlockwiseSpMatrix().init_random(1024, 96, 32, 1, 0.5, True, 42, values="uniform")
    last = sb.BlockwiseSpMatrix().init_random(256, 1024, 64, 1, 0.3, True, 43, values="uniform")
    for m in (first, layer, last):
        m.transform_and_sync_device()
    bias = dev(sb.uniform_half(44, 1024))
    x = [dev(sb.uniform_half(50 + i, K * 96).reshape(K, 96)) for i in range(8)]
    y1 = torch.zeros(tokens, 96, dtype=torch.float16, device="cuda")                                  # read on as 64 tokens of 96
    y2 = torch.zeros(1024, tokens, dtype=torch.float16, device="cuda")
    stream = torch.cuda.current_stream()

    def run(wait):
        out = [torch.zeros(256, tokens, dtype=torch.float16, device="cuda") for _ in x]
        ops = [(sb.SpmmBlockwiseOp().initialize(first, 96, a, 0.0625, None, 0.0, y1),
                sb.SpmmBlockwiseOp().initialize(last, tokens, y2, 0.0625, None, 0.0, y3)) for a, y3 in zip(x, out)]
        torch.cuda.synchronize()
        for before, behind in ops:
            before(stream)
            wait()
            assert bw.linear_direct(layer, tokens, y1, bias, tokens, y2, stream)
            wait()
            behind(stream)
            wait()
        torch.cuda.synchronize()
        return out

    want = run(torch.cuda.synchronize)
    assert all(torch.isfinite(w).all() and w.abs().max() > 0 for w in want) and not torch.equal(want[0], want[1])
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(run(lambda: None), want))
    for m in (first, layer, last):
        m.device_status()


SPECIAL = np.array([np.inf, -np.inf, np.nan, 65504, -65504, -0.0, 6e-8, 0], np.float16)


def _same(a, b):
    """Equal bits, any NaN equal to any other."""
    return bool(((a.view(torch.int16) == b.view(torch.int16)) | (a.isnan() & b.isnan())).all())


@pytest.mark.parametrize("V,permute,density", [(64, True, 0.3), (64, False, 0.9), (32, True, 0.3), (32, False, 0.3), (128, True, 0.9)])
def test_special_values_of_a_bias(V, permute, density):
    bias = dev(np.resize(SPECIAL, 256))
    lin = ShflBWLinear(sb.BlockwiseSpMatrix().init_random(256, 320, V, 1, density, permute, 31, values="uniform"), bias).cuda()
    conv = ShflBWConv2d(sb.BlockwiseSpFilter().init_random(256, 1, 1, 64, V, 1, density, permute, 32, values="uniform"), 1, bias).cuda()
    x = dev(sb.uniform_half(33, 80 * 320).reshape(80, 320))
    xc = dev(sb.uniform_half(34, 3 * 5 * 5 * 64).reshape(3, 5, 5, 64)).permute(0, 3, 1, 2)
    for module, inp, shape in ((lin, x, (1, 256)), (conv, xc, (1, 256, 1, 1))):
        y = module(inp)
        module.bias = None
        want = module(inp) + bias.reshape(shape)
        module.bias = bias
        torch.cuda.synchronize()
        assert y.isnan().any() and y.isinf().any() and _same(y.contiguous(), want.contiguous())


def test_block_columns_through_the_linear_layer():
    m = sb.BlockwiseSpMatrix().init_random(256, 320, 64, 4, 0.3, True, 41, values="uniform")
    bias = dev(sb.uniform_half(42, 256))
    lin = ShflBWLinear(m, bias).cuda()
    x = dev(sb.uniform_half(43, 37 * 320).reshape(37, 320))
    y = lin(x)
    want = x.double() @ lin.dense_weight().to("cuda").double().t() + bias.double()
    torch.cuda.synchronize()
    m.device_status()
    # the product and the sum are rounded to fp16 once each; the product is at most |want| + 1
    assert ((y.double() - want).abs() <= 2.0 ** -10 * (want.abs() + 1)).all()
