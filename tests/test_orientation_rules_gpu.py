"""Which kernel a layer takes by its depth, height and size: either orientation and either gather add the same columns in the
same order, so that every choice gives the bits of the others."""
import numpy as np
import pytest
import torch

import shflbw_sparse_nn_b200 as sb
from gpu_util import dev, host, operand_swap

pytestmark = pytest.mark.gpu


def _chained(f, Bn, H, R, stride, R_next, residual, swap, gather, monkeypatch):
    if gather is None:
        monkeypatch.delenv("SHFLBW_GATHER", raising=False)
    else:
        monkeypatch.setenv("SHFLBW_GATHER", str(gather))
    Ho = -(-H // stride)
    x = dev(sb.uniform_half(3, sb.chain_buffer_elems(f.C, H, H, Bn, R, R)))
    n = sb.chain_buffer_elems(f.F, Ho, Ho, Bn, R_next, R_next)
    out, res = torch.zeros(n, dtype=torch.float16, device="cuda"), dev(sb.uniform_half(4, n))
    with operand_swap(swap):
        op = sb.SpconvChainOp().initialize(f, Bn, H, H, stride, x, out, R_next, R_next, alpha=0.25, relu=True)
        if residual:
            op.set_residual(res, None)
    op(torch.cuda.current_stream())
    torch.cuda.synchronize()
    f.device_status()
    return host(out).view(np.uint16).copy(), op._state


@pytest.mark.parametrize("V,Bn,H,Cc,R,stride,R_next,cols,variant,gather", [
    (64, 64, 14, 128, 3, 1, 1, 230, 0, 1),      # deep: tokens in lanes all the same
    (64, 8, 15, 128, 3, 1, 1, 230, 0, 1),       # ... of padded rows
    (64, 8, 15, 128, 3, 1, 3, 230, 1, 1),       # ... into a halo: rows
    (64, 8, 5, 128, 3, 1, 1, 230, 1, 1),        # a handful of items: rows
    (64, 64, 14, 256, 3, 1, 1, 1300, 1, 1),     # the MMAs bound it: rows
    (128, 64, 14, 256, 3, 1, 1, 1300, 0, 1),
    (128, 64, 14, 128, 1, 1, 3, 20, 0, 1),
    (128, 64, 14, 128, 1, 1, 1, 100, 0, 0),     # a stage and a half
    (128, 64, 14, 256, 1, 1, 1, 150, 0, 1),
    (128, 24, 13, 128, 3, 1, 1, 150, 0, 0),     # padded rows
    (128, 8, 7, 256, 1, 1, 1, 20, 0, 1),        # fewer items than SMs, 128-token tiles
    (128, 64, 14, 64, 3, 2, 1, 230, 0, 1),      # strided, a box per pixel
])
@pytest.mark.parametrize("residual", [False, True])
def test_chained_layers(V, Bn, H, Cc, R, stride, R_next, cols, variant, gather, residual, monkeypatch):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the item counts are of 148 SMs")
    F = V * (4 if Bn * H < 60 else 10)
    f = sb.BlockwiseSpFilter().init_random(F, R, R, Cc, V, 1, (cols + 0.5) / (R * R * Cc), True, 5, values="uniform")
    f.transform_and_sync_device()
    got, st = _chained(f, Bn, H, R, stride, R_next, residual, None, None, monkeypatch)
    assert (st.variant, st.gather) == (variant, gather)
    for swap in (0, 1):
        other, st = _chained(f, Bn, H, R, stride, R_next, residual, swap, 0, monkeypatch)
        assert (st.variant, st.gather) == (swap, 0)
        assert np.array_equal(got, other)
    assert np.abs(got.view(np.float16).astype(np.float32)).max() > 0
