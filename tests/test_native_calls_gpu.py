"""The native host path of a call: the same results, strides and errors as the Python code behind it, and nothing taken from
calls that are not plain (subclasses, transforms, modes, gradients to record, other layouts and types)."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from torch import nn                                                     # noqa: E402

from shflbw_sparse_nn_b200 import _cabi, blockwise as bw                 # noqa: E402
from shflbw_sparse_nn_b200.nn import ShflBWConv2d, ShflBWLinear          # noqa: E402

pytestmark = pytest.mark.gpu


class Sub(torch.Tensor):
    pass


def _raw(module, x):
    n = _cabi.native()
    if isinstance(module, ShflBWLinear):
        return n.linear(x, module.bias, module.spmat._h.value, module.in_features, module.out_features)
    return n.conv2d(x, module.bias, module.spfilter._h.value, module.stride, module.in_channels, module.out_channels)


def _python(monkeypatch, module, x):
    with monkeypatch.context() as m:
        m.setattr(_cabi, "native", lambda: None)
        return module(x)


def _linear(bias=True):
    torch.manual_seed(1)
    return ShflBWLinear.from_dense(nn.Linear(192, 128, bias=bias), V=32, density=0.25).cuda()


def _conv(bias=True):
    torch.manual_seed(2)
    return ShflBWConv2d.from_dense(nn.Conv2d(16, 64, 3, 2, 1, bias=bias), V=32, density=0.3).cuda()


def _same(a, b):
    return a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.parametrize("bias", (False, True))
@pytest.mark.parametrize("tokens", (1, 7, 8, 37, 300))
def test_linear_as_in_python(monkeypatch, tokens, bias):
    lin = _linear(bias)
    x = torch.randn(tokens, 192, device="cuda").half()
    want = _python(monkeypatch, lin, x)
    assert _same(_raw(lin, x), want) and _same(lin(x), want)


@pytest.mark.parametrize("bias", (False, True))
@pytest.mark.parametrize("shape", ((1, 16, 1, 1), (2, 16, 7, 9), (3, 16, 14, 14)))
def test_conv_as_in_python(monkeypatch, shape, bias):
    conv = _conv(bias)
    x = torch.randn(*shape, device="cuda").half().to(memory_format=torch.channels_last)
    want = _python(monkeypatch, conv, x)
    assert _same(_raw(conv, x), want) and _same(conv(x), want)


@pytest.mark.parametrize("make", (_linear, _conv))
def test_what_is_not_plain_stays_with_python(monkeypatch, make):
    module = make()
    x = torch.randn(8, 192, device="cuda").half() if make is _linear \
        else torch.randn(2, 16, 6, 6, device="cuda").half().to(memory_format=torch.channels_last)
    assert _raw(module, x) is None                                       # not uploaded yet
    want = module(x)
    assert _same(_raw(module, x), want)
    assert _raw(module, x.as_subclass(Sub)) is None
    assert _raw(module, x.float()) is None and _raw(module, x.cpu()) is None
    assert _raw(module, torch._neg_view(x)) is None
    assert _raw(module, x[:0]) is None
    assert _raw(module, torch.cat((x, x), 1)[:, :x.shape[1]]) is None    # strides
    assert _raw(module, None) is None
    with torch.device("cuda"):                                           # a torch-function mode
        assert _raw(module, x) is None
    seen = []
    torch.func.vmap(lambda t: (seen.append((_raw(module, t), _raw(module, x))), t)[1])(x[None])
    assert seen == [(None, None)]
    torch.jit.trace(lambda t: (seen.append(_raw(module, t)), t * 2)[1], (x,), check_trace=False)
    assert seen[1:] and all(s is None for s in seen[1:])
    other = copy.copy(module)
    other._buffers = dict(module._buffers)
    for b in (module.bias.float(), module.bias[:-1], torch.stack((module.bias, module.bias), 1)[:, 0],
              module.bias.clone().requires_grad_(), module.bias.cpu(), torch._neg_view(module.bias), 3):
        other._buffers["bias"] = b
        assert _raw(other, x) is None
    with torch.no_grad():
        other._buffers["bias"] = module.bias.clone().requires_grad_()
        assert _same(_raw(other, x), want)
    with torch.autograd.forward_ad.dual_level():
        other._buffers["bias"] = torch.autograd.forward_ad.make_dual(module.bias, torch.ones_like(module.bias))
        assert _raw(other, x) is None
    with pytest.raises((TypeError, ValueError)):
        module(x.float())


def test_operators_take_every_stream_form(monkeypatch):
    m = bw.BlockwiseSpMatrix().init_random(64, 64, 16, 1, 0.3, True, 3, values="uniform")
    m.transform_and_sync_device()
    N = 40
    b = torch.randn(m.ncol, N, device="cuda").half()
    d = [torch.zeros(m.nrow, N, dtype=torch.float16, device="cuda") for _ in range(2)]
    ops = [bw.SpmmBlockwiseOp().initialize(m, N, b, t) for t in d]
    with monkeypatch.context() as p:
        p.setattr(_cabi, "native", lambda: None)
        ops[0](None)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for stream in (None, 0, side, side.cuda_stream, np.int64(side.cuda_stream)):
        d[1].zero_()
        torch.cuda.synchronize()
        ops[1](stream)
        torch.cuda.synchronize()
        assert torch.equal(*d)
    with pytest.raises((TypeError, ValueError)):
        ops[1]("no stream")
    with pytest.raises(Exception):
        bw.SpmmBlockwiseOp()(None)                                       # a state that no init has filled


@pytest.mark.parametrize("stride", (0, -1, 2 ** 31, 2 ** 32 + 1))
def test_a_stride_that_is_none_stays_with_python(stride):
    """A division by it would end the process; as 32 bits it may be another one."""
    conv = _conv()
    x = torch.randn(2, 16, 6, 6, device="cuda").half().to(memory_format=torch.channels_last)
    conv(x)                                                              # uploads the filter
    conv.stride = stride
    assert _raw(conv, x) is None
    if stride <= 0:
        with pytest.raises(Exception):                                   # ZeroDivisionError, an extent below zero
            conv(x)
