"""torch.nn front end: prune a trained `nn.Linear` / `nn.Conv2d` to Shfl-BW and run it through
the library's C ABI on the caller's CUDA stream.

    lin  = ShflBWLinear.from_dense(dense_linear, V=64, density=0.1)     # y = lin(x)
    conv = ShflBWConv2d.from_dense(dense_conv, V=64, density=0.2)       # y = conv(x)

The reference project has no such layer (it only ever builds random patterns,
block_sparse/spmm/blockwise_format.h:70-123, and points to the paper for real models); this
is the piece a user with a trained network needs in front of the hot path.  torch is the
plumbing here (device buffers, the current stream, layout views, and the inputs and biases that a
kernel cannot read where they are); pruning is `pruner.prune_matrix` / `prune_conv_filter` on the
host, once, and every forward is the library's SpMM / SpConv kernels, which add the bias too.  fp16
inference only; there is no backward pass through the product.
"""
from __future__ import annotations

from contextlib import nullcontext

import numpy as np
import torch
from torch import nn
from torch.autograd import forward_ad

from . import _cabi, blockwise as bw
from .pruner import prune_conv_filter, prune_matrix


_NOTHING = nullcontext()


def _require_cuda_half(x: torch.Tensor, what: str):
    if not x.is_cuda or x.dtype != torch.float16:
        raise TypeError(f"{what}: expected a CUDA float16 tensor, got {x.device} {x.dtype}")


def _on_device(device: torch.device):
    """Makes `device` current where it is not."""
    return _NOTHING if device.index == torch.cuda.current_device() else torch.cuda.device(device)


def _stream_of(device: torch.device) -> int:
    """torch's current stream on `device` as a cudaStream_t (without building a Stream object, 3 us)."""
    return torch._C._cuda_getCurrentRawStream(device.index)


def _bias_of(module: nn.Module):
    """module.bias, without torch's look through its dictionaries where it is the buffer that it was made as."""
    return module._buffers["bias"] if "bias" in module._buffers else module.bias


def _in_memory(x: torch.Tensor) -> bool:
    """Whether x.data_ptr() addresses the values of `x`: not where a negation is still pending (the memory
    holds -x) and not for a tensor without memory of its own (a wrapper subclass, whose pointer is 0)."""
    return not x.is_neg() and x.data_ptr() != 0


def _carries_gradient(t: torch.Tensor) -> bool:
    """Whether an operation of torch on `t` would record a gradient or carry a tangent along."""
    if t.requires_grad and torch.is_grad_enabled():
        return True
    return forward_ad._current_level >= 0 and forward_ad.unpack_dual(t).tangent is not None


def _fused_bias(bias, device: torch.device, n: int, align: int):
    """(bias on `device`, whether the kernels can add it: fp16, one per output, contiguous, aligned, its values
    in memory and without a gradient to record).  Every other bias is added by torch."""
    if bias is None:
        return None, False
    if bias.device != device:
        bias = bias.to(device)
    fused = bias.dtype == torch.float16 and bias.shape == (n,) and bias.is_contiguous() and not bias.is_neg() \
        and not _carries_gradient(bias)
    if fused:
        address = bias.data_ptr()
        fused = address != 0 and address % align == 0        # (0: as in _in_memory)
    return bias, fused


class ShflBWLinear(nn.Module):
    """y = x @ W_pruned^T + b with W in the Shfl-BW format.

    The SpMM computes D[out][tokens] = A[out][in] . B[in][tokens], i.e. it wants activations
    feature-major (tokens contiguous).  `forward` takes the usual [..., in_features] tensor,
    pays one transpose kernel and returns a view of the feature-major result;
    `forward_feature_major` takes [in_features][tokens] and returns [out_features][tokens] with no
    copies (tokens a multiple of 8).  The bias is added in the SpMM kernel."""

    def __init__(self, spmat: bw.BlockwiseSpMatrix, bias: torch.Tensor | None, info: dict | None = None):
        super().__init__()
        self.spmat = spmat
        self.in_features, self.out_features = spmat.ncol, spmat.nrow
        self.info = info or {}
        self.register_buffer("bias", None if bias is None else bias.detach().to(torch.float16))
        self._uploaded_on = None

    @classmethod
    def from_dense(cls, linear: nn.Linear, V: int = 64, density: float = 0.1, permute: bool = True, seed=None):
        m, info = prune_matrix(linear.weight.detach().float().cpu().numpy(), V, density, permute, seed=seed)
        return cls(m, linear.bias, info)

    def _upload(self, device: torch.device):
        if self._uploaded_on != device:
            with torch.cuda.device(device):
                self.spmat.transform_and_sync_device()
            self._uploaded_on = device

    def _run(self, x, tokens: int, xt, n: int) -> torch.Tensor:
        """out[M][n] = W . xt + bias; x (token-major, or None when xt holds the operand) is read as it is, or transposed first."""
        dev = xt.device if x is None else x.device
        self._upload(dev)
        out = torch.empty((self.out_features, n), dtype=torch.float16, device=dev)
        bias, fused = _fused_bias(self.bias, dev, self.out_features, 2)
        with _on_device(dev):
            added, stream = bias if fused else None, _stream_of(dev)
            if x is None or not bw.linear_direct(self.spmat, tokens, x, added, n, out, stream):
                if xt is None:
                    xt = torch.empty((self.in_features, n), dtype=torch.float16, device=dev)
                bw.linear_exec(self.spmat, tokens, x, added, xt, n, out, stream)
        if bias is not None and not fused:
            out += bias[:, None]
        return out

    def forward_feature_major(self, xt: torch.Tensor) -> torch.Tensor:
        _require_cuda_half(xt, "ShflBWLinear")
        if xt.dim() != 2 or xt.shape[0] != self.in_features or xt.shape[1] % 8 or not xt.is_contiguous():
            raise ValueError("expected a contiguous [in_features][tokens] tensor with tokens % 8 == 0")
        xt = xt.resolve_neg()
        return self._run(None, xt.shape[1], xt, xt.shape[1])

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        native = _cabi.native()
        if native is not None:                               # plain operands: everything below as one native call
            spmat = self.spmat                               # (held: the call has its address only, and lets other threads run)
            y = native.linear(x, _bias_of(self), spmat._h.value or 0, self.in_features, self.out_features)
            if y is not None:
                return y
        _require_cuda_half(x, "ShflBWLinear")
        shape = x.shape
        x2 = x if len(shape) == 2 and shape[1] == self.in_features else x.reshape(-1, self.in_features)
        tokens = x2.shape[0]
        padded = -(-tokens // 8) * 8
        # Tokens in consecutive memory (the view that a layer like this one returns) are in the operand's order
        # already: one plain copy by torch.  4096 x 4096 at density 0.1, 4096 tokens, the whole call on the device:
        # 45 us; made contiguous and then transposed by the kernel, as every other order is, 110.  A ragged count
        # needs a fill and a slice as well, 5 us of host time, and gains from a few million values on (4095 tokens:
        # 78 us against 110).
        by_torch = False
        if not x2.is_contiguous():
            by_torch = x2.stride(0) == 1 and (tokens == padded or x2.numel() >= 1 << 22)
            if not by_torch:
                x2 = x2.contiguous()
        if tokens and not _in_memory(x2):                    # the kernel cannot read it
            by_torch = True
        xt = None
        if by_torch:
            xt = (torch.empty if tokens == padded else torch.zeros)((self.in_features, padded), dtype=torch.float16, device=x.device)
            (xt if tokens == padded else xt[:, :tokens]).copy_(x2.t())
            x2 = None
        yt = self._run(x2, tokens, xt, padded)
        y = yt.as_strided((tokens, self.out_features), (1, padded))
        return y if len(shape) == 2 and shape[0] == tokens else y.reshape(*shape[:-1], self.out_features)

    def dense_weight(self) -> torch.Tensor:
        """The pruned weights as a dense [out][in] fp16 tensor (rows in original order), for checks."""
        return torch.from_numpy(densify(self.spmat))


class ShflBWConv2d(nn.Module):
    """Conv2d with a Shfl-BW filter: square odd kernel, padding = kernel // 2, equal strides,
    no dilation or groups, in_channels % 8 == 0, out_channels % V == 0.  Input and output are
    NCHW tensors as torch modules exchange them; channels-last memory format makes both sides
    zero-copy views of the NHWC buffers the kernel reads and writes."""

    def __init__(self, spfilter: bw.BlockwiseSpFilter, stride: int, bias: torch.Tensor | None, info: dict | None = None):
        super().__init__()
        self.spfilter, self.stride = spfilter, int(stride)
        self.in_channels, self.out_channels, self.kernel_size = spfilter.C, spfilter.F, spfilter.R
        self.info = info or {}
        self.register_buffer("bias", None if bias is None else bias.detach().to(torch.float16))
        self._uploaded_on = None

    @classmethod
    def from_dense(cls, conv: nn.Conv2d, V: int = 64, density: float = 0.2, permute: bool = True, seed=None):
        kh, kw = conv.kernel_size
        if kh != kw or kh % 2 == 0 or conv.padding not in ((kh // 2, kh // 2), kh // 2) or conv.dilation not in ((1, 1), 1) \
                or conv.groups != 1 or conv.stride[0] != conv.stride[1] or conv.padding_mode != "zeros":
            raise ValueError("ShflBWConv2d: square odd kernel, padding = kernel // 2, equal strides, no dilation / groups")
        if conv.in_channels % 8:
            raise ValueError("ShflBWConv2d: in_channels must be a multiple of 8")
        f, info = prune_conv_filter(conv.weight.detach().float().cpu().numpy(), V, density, permute, seed=seed)
        return cls(f, conv.stride[0], conv.bias, info)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        native = _cabi.native()
        if native is not None:                               # plain operands: everything below as one native call
            spfilter = self.spfilter                         # (held, as above)
            y = native.conv2d(x, _bias_of(self), spfilter._h.value or 0, self.stride, self.in_channels, self.out_channels)
            if y is not None:
                return y
        _require_cuda_half(x, "ShflBWConv2d")
        if x.dim() != 4 or x.shape[1] != self.in_channels:
            raise ValueError(f"expected [N][{self.in_channels}][H][W]")
        if self._uploaded_on != x.device:
            with torch.cuda.device(x.device):
                self.spfilter.transform_and_sync_device()
            self._uploaded_on = x.device
        n, _, h, w = x.shape
        x_nhwc = x.permute(0, 2, 3, 1).contiguous().resolve_neg()   # a view when x is channels-last
        ho, wo = -(-h // self.stride), -(-w // self.stride)
        out = torch.empty((n, ho, wo, self.out_channels), dtype=torch.float16, device=x.device)
        bias, fused = _fused_bias(self.bias, x.device, self.out_channels, 16)
        with _on_device(x.device):
            op = bw.SpconvBlockwiseOp().initialize(self.spfilter, n, h, w, self.stride, x_nhwc, out)
            op.run_with_bias(bias if fused else None, _stream_of(x.device))
        if bias is not None and not fused:
            out += bias
        return out.permute(0, 3, 1, 2)                       # NCHW view of the NHWC result (channels-last)

    def dense_weight(self) -> torch.Tensor:
        """The pruned filter as a dense [F][C][R][S] fp16 tensor, for checks."""
        d = densify(self.spfilter).reshape(self.out_channels, self.kernel_size, self.kernel_size, self.in_channels)
        return torch.from_numpy(np.ascontiguousarray(d.transpose(0, 3, 1, 2)))


def densify(m) -> np.ndarray:
    """Logical dense matrix (rows in original order) of a Shfl-BW object, fp16."""
    d = np.zeros((m.nrow, m.ncol), np.float16)
    v = np.asarray(m.values).view(np.float16).reshape(-1, m.brow)   # one row per stored column
    perm = m.row_permute_ids if m.row_permute else np.arange(m.nrow)
    bcol = m.bcol
    indptr = m.indptr * bcol
    indices = (m.indices[:, None] * bcol + np.arange(bcol)[None, :]).reshape(-1)
    for i in range(m.nrow // m.brow):
        rows = perm[i * m.brow:(i + 1) * m.brow]
        cols = indices[indptr[i]:indptr[i + 1]]
        d[np.ix_(rows, cols)] = v[indptr[i]:indptr[i + 1]].T
    return d
