"""The one-launch linear layer on a few tokens: the bits of the two launches and their distance from 64-bit sums, at the edges of its tiles (tokens of a block, columns of a
pass, rows of a block), on unaligned and odd rows; the rule that sends calls to it; nothing read beyond the tokens."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from torch import nn                                                     # noqa: E402

import shflbw_sparse_nn_b200 as sb                                        # noqa: E402
from shflbw_sparse_nn_b200 import blockwise as bw                         # noqa: E402
from shflbw_sparse_nn_b200.nn import ShflBWLinear, densify                # noqa: E402

pytestmark = pytest.mark.gpu


def _matrix(V, K, per, permute, seed=0):
    rng = np.random.default_rng(seed)
    indptr = np.concatenate(([0], np.cumsum(per))).astype(np.int32)
    indices = np.concatenate([np.sort(rng.choice(K, n, replace=False)) for n in per]).astype(np.int32)
    values = (rng.random((indptr[-1], V)) * 2 - 1).astype(np.float16)
    perm = rng.permutation(V * len(per)).astype(np.int32) if permute else None
    m = sb.BlockwiseSpMatrix.from_arrays(V * len(per), K, V, indptr, indices, values.view(np.uint16).reshape(-1), perm)
    m.transform_and_sync_device()
    return m


@pytest.mark.parametrize("V", (16, 32, 64, 128))
@pytest.mark.parametrize("tokens", (1, 7, 8, 9, 37))
@pytest.mark.parametrize("K,per", ((1303, (1, 16, 17, 511, 512, 513, 1303, 0)), (24, (24, 0, 3))))
def test_against_64_bits(monkeypatch, V, tokens, K, per):
    monkeypatch.setenv("SHFLBW_LINEAR_DIRECT", "1")
    m = _matrix(V, K, per, permute=V != 32, seed=V + tokens)
    M, N = m.nrow, -(-tokens // 8) * 8
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    dense = torch.from_numpy(densify(m)).cuda().double()
    for bias in (None, (torch.rand(M, generator=gen, device="cuda") * 2 - 1).half()):
        buf = torch.full((tokens * K + 2 * K,), float("nan"), dtype=torch.float16, device="cuda")      # x amid NaN, 2-byte aligned
        x = buf[K:K + tokens * K].view(tokens, K)
        x.copy_(torch.rand(tokens, K, generator=gen, device="cuda") * 2 - 1)
        out = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        assert bw.linear_direct(m, tokens, x, bias, N, out, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want = dense @ x.double().t()
        # 32-bit sums of n products in any order, n * 2^-23 * sum |a b| (sums chopped, not rounded), and a rounding to fp16 ...
        n = max(max(per), 1)
        bound = n * 2.0 ** -23 * (dense.abs() @ x.double().abs().t()) + want.abs() * 2.0 ** -11 + 2.0 ** -25
        if bias is not None:                                              # ... and another one with the bias added
            want = want + bias.double()[:, None]
            bound = bound + (want.abs() + bound) * 2.0 ** -11 + 2.0 ** -25
        assert bool(((out[:, :tokens].double() - want).abs() <= bound).all())
        pad = out[:, tokens:]
        xt = torch.empty(K, N, dtype=torch.float16, device="cuda")
        other = torch.empty_like(out)
        bw.linear_exec(m, tokens, x, bias, xt, N, other, torch.cuda.current_stream())
        assert torch.equal(out.view(torch.int16), other.view(torch.int16))
        assert torch.equal(pad, (bias if bias is not None else torch.zeros(M, device="cuda").half())[:, None].expand_as(pad))


@pytest.mark.parametrize("scale", (1e-6, 6e4, float("inf")))
def test_values_at_the_ends_of_the_range(monkeypatch, scale):
    monkeypatch.setenv("SHFLBW_LINEAR_DIRECT", "1")
    m = _matrix(32, 200, (40, 200, 7), True)
    x = (torch.rand(11, 200, device="cuda") * 2 - 1)
    x = torch.where(torch.rand(11, 200, device="cuda") < 0.02, torch.tensor(scale, device="cuda"), x * min(scale, 1.0)).half()
    bias = torch.full((m.nrow,), -1.0, device="cuda").half()
    xt, a, b = (torch.empty(r, 16, dtype=torch.float16, device="cuda") for r in (200, m.nrow, m.nrow))
    bw.linear_exec(m, 11, x, bias, xt, 16, a, torch.cuda.current_stream())
    assert bw.linear_direct(m, 11, x, bias, 16, b, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(nan=0.5), b.nan_to_num(nan=0.5))


def test_rule_and_module():
    m = _matrix(64, 2048, (205,) * 32, True)
    go = lambda tokens: bw.linear_direct(m, tokens, torch.zeros(tokens, 2048, device="cuda").half(), None, -(-tokens // 8) * 8,
                                         torch.empty(2048, -(-tokens // 8) * 8, dtype=torch.float16, device="cuda"))
    assert go(1) and go(8) and go(37) and not go(1000)
    lin = ShflBWLinear(m, (torch.rand(2048) * 2 - 1)).cuda()
    w = lin.dense_weight().cuda().float()
    for tokens in (5, 1000):                                              # each side of the rule
        x = (torch.rand(tokens, 2048, device="cuda") * 2 - 1).half()
        want = x.float() @ w.t() + lin.bias.float()
        assert float((lin(x).float() - want).abs().max()) <= float(want.abs().max()) * 2.0 ** -10 + 205 * 205 * 2.0 ** -23
    odd = sb.BlockwiseSpMatrix().init_random(48, 64, 24, 1, 0.3, False, 3, values="uniform")   # no tensor-core kernel has such blocks
    odd.transform_and_sync_device()
    x = torch.zeros(8, 64, device="cuda").half()
    assert not bw.linear_direct(odd, 8, x, None, 8, torch.empty(48, 8, dtype=torch.float16, device="cuda"))
    with pytest.raises(Exception):
        bw.linear_direct(m, 0, x, None, 8, x)


class _Ints:
    """Device memory as a tensor."""
    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (address, False), "version": 3}


def test_ids_outside_the_layer_read_nothing_outside_x(monkeypatch):
    """The ids lie in device memory: whatever stands there, the reads stay in x.  Beyond the last column they read that one, as
    the panel kernel's do; negative ones read nothing."""
    monkeypatch.setenv("SHFLBW_LINEAR_DIRECT", "1")
    K, tokens, N = 96, 11, 16
    m = _matrix(32, K, (40, 96), True)
    x = (torch.rand(tokens, K, device="cuda") * 2 - 1).half()
    out = [torch.full((m.nrow, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2)]
    op = sb.SpmmBlockwiseOp().initialize(m, N, torch.zeros(K, N, device="cuda").half(), out[0])
    ids = torch.as_tensor(_Ints(op._state.blk_idx, 48 + 96), device="cuda")
    at = torch.tensor([0, 7, 39, 47, 48, 143], device="cuda")
    for bad in ([K, K + 5, 2 ** 31 - 1, 1 << 20, K, K], [-1, -2 ** 31, -K, -2, -1, -1]):
        if bad[0] < 0:
            x[:, K - 1] = 0
        for y, there in zip(out, (bad, [K - 1] * 6)):
            ids[at] = torch.tensor(there, dtype=torch.int32, device="cuda")
            assert bw.linear_direct(m, tokens, x, None, N, y, torch.cuda.current_stream())
            torch.cuda.synchronize()
        assert torch.equal(*out) and not out[0].isnan().any()
