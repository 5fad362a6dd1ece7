"""Permuted filters whose small outputs the panel kernel puts in order by itself: the bits of the same call with a pass behind
it, with and without a bias, over block heights, ragged batches and images, and images beyond the batch; the rule's two sides."""
import pytest

torch = pytest.importorskip("torch")
import shflbw_sparse_nn_b200 as sb                                        # noqa: E402

pytestmark = pytest.mark.gpu


def _call(f, shape, stride, bias, launches=None):
    B, H, W, _ = shape
    x = (torch.rand(shape, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") * 2 - 1).half()
    n = B * -(-H // stride) * -(-W // stride) * f.F
    buf = torch.full((n + 2 * f.F,), float("nan"), dtype=torch.float16, device="cuda")      # nothing beside the output is written
    y = buf[f.F:f.F + n]
    op = sb.SpconvBlockwiseOp().initialize(f, B, H, W, stride, x, y)
    assert launches is None or op.launches_per_exec == launches
    op.run_with_bias(bias)
    torch.cuda.synchronize()
    assert buf[:f.F].isnan().all() and buf[-f.F:].isnan().all() and not y.isnan().any()
    return y.clone()


@pytest.mark.parametrize("V,F", ((16, 48), (16, 528), (32, 64), (32, 512), (64, 128), (64, 320), (128, 384)))
@pytest.mark.parametrize("shape,R,stride", (((1, 1, 1, 64), 1, 1), ((5, 27, 27, 64), 1, 2), ((9, 7, 5, 16), 3, 1), ((3, 40, 33, 24), 3, 1)))
def test_the_bits_of_the_pass(monkeypatch, V, F, shape, R, stride):
    f = sb.BlockwiseSpFilter().init_random(F, R, R, shape[3], V, 1, 0.3, True, 5, values="uniform")
    f.transform_and_sync_device()
    for bias in (None, (torch.rand(F, device="cuda") * 2 - 1).half()):
        got = []
        for scatter, launches in (("0", 3), ("1", 2)):
            monkeypatch.setenv("SHFLBW_CONV_SCATTER", scatter)
            monkeypatch.setenv("SHFLBW_CONV_PLANES", "0")
            got.append(_call(f, shape, stride, bias, launches))
        assert torch.equal(*got)


def test_rule():
    for shape, F, V, launches in (((5, 27, 27, 256), 512, 32, 2), ((24, 17, 17, 128), 256, 64, 3), ((40, 20, 20, 64), 640, 32, 3)):
        f = sb.BlockwiseSpFilter().init_random(F, 1, 1, shape[3], V, 1, 0.1, True, 5, values="uniform")
        f.transform_and_sync_device()
        _call(f, shape, 2 if shape[0] == 5 else 1, None, launches)


@pytest.mark.parametrize("shape,F,V,stride,launches", (
    ((5, 12, 12, 32), 512, 64, 2, 3), ((11, 13, 13, 16), 320, 64, 2, 3),   # 24 and 35 items of 2450 sectors: the pass has all SMs
    ((4, 13, 13, 416), 384, 64, 2, 2), ((5, 27, 27, 256), 512, 32, 2, 2)))  # 24 of 1750; 208 items, two rounds of 2858
def test_few_items_scatter_less(shape, F, V, stride, launches):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shares are of 148 SMs")
    f = sb.BlockwiseSpFilter().init_random(F, 1, 1, shape[3], V, 1, 0.25, True, 5, values="uniform")
    f.transform_and_sync_device()
    _call(f, shape, stride, None, launches)
