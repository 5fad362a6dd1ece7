"""Filters whose permutation moves rows only within their blocks: NHWC calls need no pass behind the panel kernel, and
give the bits of the same filter stored in logical order; a permutation across blocks still takes that pass."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import shflbw_sparse_nn_b200 as sb                                        # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,blocks,R,stride,shape", (
    (16, 1, 1, 1, (1, 5, 3, 24)), (32, 1, 3, 1, (5, 9, 7, 16)), (64, 1, 3, 1, (32, 56, 56, 64)), (128, 1, 3, 2, (9, 13, 13, 64)),
    (64, 3, 3, 1, (16, 14, 14, 64)), (16, 4, 1, 2, (3, 11, 11, 40))))
def test_rows_within_blocks(monkeypatch, V, blocks, R, stride, shape):
    B, H, W, Cn = shape
    F, K = V * blocks, R * R * Cn
    rng = np.random.default_rng(V + blocks)
    per = [min(K, n) for n in (K // 3 + 1, 0, K, 1)[:blocks]]             # an empty block among them
    indptr = np.concatenate(([0], np.cumsum(per))).astype(np.int32)
    indices = np.concatenate([np.sort(rng.choice(K, n, replace=False)) for n in per]).astype(np.int32)
    values = (rng.random((indptr[-1], V)) * 2 - 1).astype(np.float16)
    local = [rng.permutation(V) for _ in range(blocks)]
    logical = np.zeros_like(values)                                       # the same filter with its rows in logical order
    for i, p in enumerate(local):
        logical[indptr[i]:indptr[i + 1], p] = values[indptr[i]:indptr[i + 1]]
    perm = np.concatenate([i * V + p for i, p in enumerate(local)]).astype(np.int32)
    make = lambda vals, ids: sb.BlockwiseSpFilter.from_arrays(F, R, R, Cn, V, indptr, indices, vals.view(np.uint16).reshape(-1), ids)
    x = (torch.rand(shape, device="cuda") * 2 - 1).half()
    Ho, Wo = -(-H // stride), -(-W // stride)
    bias = (torch.rand(F, device="cuda") * 2 - 1).half()
    got = []
    for f in (make(values, perm), make(logical, None)):
        f.transform_and_sync_device()
        y = [torch.full((B, Ho, Wo, F), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2)]
        for b, out in zip((None, bias), y):
            op = sb.SpconvBlockwiseOp().initialize(f, B, H, W, stride, x, out)
            assert op.launches_per_exec == 2
            op.run_with_bias(b)
        torch.cuda.synchronize()
        got += [y]
    assert all(torch.equal(a, b) for a, b in zip(*got)) and not torch.isnan(got[0][0]).any()
    simt = torch.zeros((B, Ho, Wo, F), dtype=torch.float16, device="cuda")      # ... and what the CUDA-core kernel makes of it
    f = make(values, perm)
    f.transform_and_sync_device()
    sb.SpconvBlockwiseOp(sb.KERNEL_SIMT).initialize(f, B, H, W, stride, x, simt)()
    # fp32 sums of at most K products of [-1, 1): twice K * 2^-24 * sum |a b| <= K^2 * 2^-23, and one fp16 rounding each
    top = float(simt.float().abs().max())
    assert float((simt.float() - got[0][0].float()).abs().max()) <= K * K * 2.0 ** -23 + top * 2.0 ** -10
    if blocks > 1:
        across = np.roll(perm, 1)
        f = make(values, across.astype(np.int32))
        f.transform_and_sync_device()
        y = torch.empty((B, Ho, Wo, F), dtype=torch.float16, device="cuda")
        monkeypatch.setenv("SHFLBW_CONV_SCATTER", "0")
        op = sb.SpconvBlockwiseOp().initialize(f, B, H, W, stride, x, y)
        assert op.launches_per_exec == 3
        op()
        torch.cuda.synchronize()
        assert torch.equal(y[..., torch.from_numpy(across).long().cuda()], got[0][0][..., torch.from_numpy(perm).long().cuda()])
