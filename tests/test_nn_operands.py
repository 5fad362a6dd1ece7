"""Which tensors the module front end hands to the kernels by address.  A kernel reads memory, so a
tensor whose memory does not hold its values (a pending negation, a wrapper subclass) or whose
addition has to be recorded by autograd must go through torch instead."""
import weakref

import pytest
import torch
from torch.autograd import forward_ad
from torch.utils._pytree import tree_map

import shflbw_sparse_nn_b200 as sb
import shflbw_sparse_nn_b200.nn as sbnn
from shflbw_sparse_nn_b200 import _cabi

CPU = torch.device("cpu")


class Wrapped(torch.Tensor):
    """A tensor without memory of its own: what is made of it is wrapped too, what reads it unwraps it."""

    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device)

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        def unwrap(a):
            return a.inner if isinstance(a, Wrapped) else a
        out = func(*tree_map(unwrap, args), **tree_map(unwrap, kwargs or {}))
        return Wrapped(out) if isinstance(args[0], Wrapped) and isinstance(out, torch.Tensor) else out


def test_bias_is_fused_only_where_the_kernel_can_read_it():
    b = torch.arange(16, dtype=torch.float16)
    assert sbnn._fused_bias(b, CPU, 16, 2) == (b, True)
    for other in (torch._neg_view(b), Wrapped(b), b.float(), b[:8], b.reshape(1, 16), torch.zeros(32, dtype=torch.float16)[::2]):
        got, fused = sbnn._fused_bias(other, CPU, 16, 2)
        assert got is other and not fused
    assert sbnn._fused_bias(None, CPU, 16, 2) == (None, False)


def test_bias_that_autograd_follows_is_not_fused():
    b = torch.ones(16, dtype=torch.float16, requires_grad=True)
    assert not sbnn._fused_bias(b, CPU, 16, 2)[1]
    with torch.no_grad():
        assert sbnn._fused_bias(b, CPU, 16, 2)[1]
    with forward_ad.dual_level():
        assert not sbnn._fused_bias(forward_ad.make_dual(torch.ones(16).half(), torch.ones(16).half()), CPU, 16, 2)[1]
        assert sbnn._fused_bias(torch.ones(16).half(), CPU, 16, 2)[1]


def test_a_native_call_holds_its_operand(monkeypatch):
    """The call gets an address and releases the GIL: what another thread then binds to the module must not free it."""
    lin = sbnn.ShflBWLinear(sb.BlockwiseSpMatrix().init_random(64, 64, 32, 1, 0.2, True, 1, values="uniform"), None)
    conv = sbnn.ShflBWConv2d(sb.BlockwiseSpFilter().init_random(64, 1, 1, 8, 32, 1, 0.5, True, 1, values="uniform"), 1, None)
    for module, name in ((lin, "spmat"), (conv, "spfilter")):
        operand = weakref.ref(getattr(module, name))
        alive = []

        class Native:
            @staticmethod
            def linear(*args):
                setattr(module, name, None)              # as another thread may meanwhile
                alive.append(operand() is not None)
                return args[0]
            conv2d = linear

        monkeypatch.setattr(_cabi, "native", lambda: Native)
        x = torch.zeros(1)
        assert module(x) is x and alive == [True] and operand() is None


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "neg", "wrapped"])
def test_modules_compute_with_the_values_of_a_tensor_and_not_its_memory(kind):
    lin = sbnn.ShflBWLinear.from_dense(torch.nn.Linear(128, 64), V=64, density=0.3).cuda()
    conv = sbnn.ShflBWConv2d.from_dense(torch.nn.Conv2d(32, 64, 1), V=64, density=0.3).cuda()
    x = (torch.rand(24, 128, device="cuda") * 2 - 1).half()
    xc = (torch.rand(3, 32, 5, 7, device="cuda") * 2 - 1).half().contiguous(memory_format=torch.channels_last)
    as_kind = {"plain": lambda t: t, "neg": lambda t: torch._neg_view(-t), "wrapped": Wrapped}[kind]
    want, want_c = lin(x), conv(xc)
    assert torch.equal(lin(as_kind(x)), want)
    if kind != "wrapped":
        xt = x.t().contiguous()
        assert torch.equal(lin.forward_feature_major(as_kind(xt)), want.t())
        assert torch.equal(conv(as_kind(xc)), want_c)
    lin._buffers["bias"], conv._buffers["bias"] = as_kind(lin.bias), as_kind(conv.bias)
    assert torch.equal(lin(x), want) and torch.equal(conv(xc), want_c)


@pytest.mark.gpu
def test_gradient_of_a_bias():
    lin = sbnn.ShflBWLinear.from_dense(torch.nn.Linear(128, 64), V=64, density=0.3).cuda()
    conv = sbnn.ShflBWConv2d.from_dense(torch.nn.Conv2d(32, 64, 1), V=64, density=0.3).cuda()
    x = (torch.rand(24, 128, device="cuda") * 2 - 1).half()
    xc = (torch.rand(3, 32, 5, 7, device="cuda") * 2 - 1).half()
    for module, inp, count in ((lin, x, 24), (conv, xc, 3 * 5 * 7)):
        want = module(inp)
        assert not want.requires_grad
        module.bias.requires_grad_()
        y = module(inp)
        assert torch.equal(y.detach(), want)
        y.float().sum().backward()
        assert torch.equal(module.bias.grad, torch.full((64,), float(count), dtype=torch.float16, device="cuda"))
