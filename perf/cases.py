"""The work that users of this framework have it do, as cases that can be timed.

Every case is fp16 inference (the only data type of the framework) with seeded random Shfl-BW
patterns, uniform[-1, 1) weights and activations, through the public entry points:

  spmm       SpmmBlockwiseOp bound once to a sparse operand and its dense buffers, one launch a pass
  spmm_host  the same product on page-locked host buffers: copies in, kernel, copies out
  linear     ShflBWLinear.forward on token-major activations, with bias
  spconv     SpconvBlockwiseOp, NHWC in and out, bound once
  conv2d     ShflBWConv2d.forward on a channels-last tensor, with bias
  resnet50   SparseResNet50: 52 chained sparse convolutions, replayed as a CUDA graph or enqueued eagerly

The forward pass is the only direction there is.  Shapes are those of the benchmark, the sweep
(`shflbw_sparse_nn_b200/sweep.py`) and the tests, or generic ones between them.
"""
import math

import numpy as np
import torch

import shflbw_sparse_nn_b200 as sb
from shflbw_sparse_nn_b200 import resnet50 as rn
from shflbw_sparse_nn_b200.nn import ShflBWConv2d, ShflBWLinear


def listed():
    return [
        # The smallest product: launch latency and nothing else.
        dict(name="spmm_256", kind="spmm", M=256, K=256, N=256, V=32, density=0.1, permute=True, alpha=1.0, beta=0.0),
        # The headline product (bench.py's default).
        dict(name="spmm_4096_v64", kind="spmm", M=4096, K=4096, N=4096, V=64, density=0.1, permute=True, alpha=1.0, beta=0.0),
        # A wide FFN projection on a short token batch, with narrow row blocks.
        dict(name="spmm_ffn_n512_v32", kind="spmm", M=11008, K=4096, N=512, V=32, density=0.25, permute=True, alpha=1.0, beta=0.0),
        # A long prefill at a mild sparsity with the tallest row blocks: the largest product.
        dict(name="spmm_prefill_v128", kind="spmm", M=4096, K=4096, N=16384, V=128, density=0.25, permute=True, alpha=1.0, beta=0.0),
        # Finest granularity, a ragged token count, no permutation, accumulating into an existing matrix.
        dict(name="spmm_ragged_v16_beta", kind="spmm", M=3072, K=768, N=1000, V=16, density=0.25, permute=False, alpha=0.5, beta=1.0),
        # The product on host buffers, end to end over the host link.
        dict(name="spmm_host_4096", kind="spmm_host", M=4096, K=4096, N=4096, V=64, density=0.1),
        # A decode step of a sparse linear layer: a handful of tokens, where latency counts.
        dict(name="linear_decode_37", kind="linear", M=4096, K=4096, tokens=37, V=64, density=0.1, permute=True, bias=True),
        # The headline convolution (bench.py's second workload).
        dict(name="spconv_14_512_2048", kind="spconv", B=16, H=14, W=14, C=512, F=2048, R=3, stride=1, V=64, density=0.1, permute=True),
        # A strided projection shortcut on an odd batch and an odd image.
        dict(name="spconv_1x1_s2_odd", kind="spconv", B=5, H=27, W=27, C=256, F=512, R=1, stride=2, V=32, density=0.2, permute=True),
        # A sparse convolution module inside a torch network, early stage: large image, few channels.
        dict(name="conv2d_56_64", kind="conv2d", B=32, H=56, W=56, C=64, F=64, R=3, stride=1, V=64, density=0.2, bias=True),
        # The whole pruned network at serving throughput, one CUDA graph a pass: the largest case.
        dict(name="resnet50_b256", kind="resnet50", B=256, H=56, V=64, density=0.2, graph=True),
        # The same network answering a small batch, enqueued launch by launch.
        dict(name="resnet50_b8", kind="resnet50", B=8, H=56, V=64, density=0.2, graph=False),
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    return max(step, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    kind = rng.choice(["spmm"] * 5 + ["linear"] * 2 + ["spconv"] * 3 + ["conv2d"] * 2 + ["resnet50", "spmm_host"])
    density = round(math.exp(rng.uniform(math.log(0.05), math.log(0.5))), 3)
    while True:
        if kind in ("spmm", "spmm_host", "linear"):
            V = rng.choice([16, 32, 64, 128]) if kind == "spmm" else rng.choice([32, 64, 128])
            c = dict(kind=kind, M=_log_int(rng, 256, 11008, V), K=_log_int(rng, 256, 4096, 8), V=V, density=density)
            if kind == "spmm":
                beta = rng.choice([0.0, 0.0, 0.0, 1.0])
                c.update(N=_log_int(rng, 8, 16384, 8), permute=rng.random() < 0.8, alpha=rng.choice([1.0, 1.0, 0.5]), beta=beta)
            elif kind == "spmm_host":
                c.update(N=_log_int(rng, 64, 8192, 8))
            else:
                c.update(tokens=_log_int(rng, 1, 4096), permute=rng.random() < 0.8, bias=rng.random() < 0.5)
        elif kind in ("spconv", "conv2d"):
            V = rng.choice([16, 32, 64, 128]) if kind == "spconv" else rng.choice([32, 64])
            c = dict(kind=kind, B=_log_int(rng, 1, 64), H=_log_int(rng, 7, 56), C=_log_int(rng, 64, 1024, 8),
                     F=_log_int(rng, 64, 2048, V), R=rng.choice([1, 3]), stride=rng.choice([1, 1, 2]), V=V, density=density)
            c["W"] = c["H"] if rng.random() < 0.7 else _log_int(rng, 7, 56)
            c.update(dict(permute=rng.random() < 0.8) if kind == "spconv" else dict(bias=rng.random() < 0.5))
        else:
            c = dict(kind=kind, B=_log_int(rng, 1, 128), H=rng.choice([32, 40, 48, 56]), V=64,
                     density=round(rng.uniform(0.1, 0.25), 3), graph=rng.random() < 0.5)
        # no dearer than the large products and the whole network
        if work(c)["flops"] <= 1.5e11 and work(c)["bytes"] <= 6e8 or kind == "resnet50":
            return c


# ------------------------------------------------------------------------------ states --

def _uniform(gen, *shape, pin=False):
    t = (torch.rand(shape, generator=gen, device="cuda") * 2 - 1).half()
    return t.cpu().pin_memory() if pin else t


def _matrix(case, seed):
    m = sb.BlockwiseSpMatrix().init_random(case["M"], case["K"], case["V"], 1, case["density"],
                                           case.get("permute", True), seed, values="uniform")
    m.transform_and_sync_device()
    return m


def _filter(case, seed):
    f = sb.BlockwiseSpFilter().init_random(case["F"], case["R"], case["R"], case["C"], case["V"], 1, case["density"],
                                           case.get("permute", True), seed, values="uniform")
    f.transform_and_sync_device()
    return f


def prepare(case, seed):
    """The sparse operand on the GPU, the activations, and the operator or module bound to them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    wseed = 1 + seed % (1 << 30)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "spmm":
        M, K, N = case["M"], case["K"], case["N"]
        s["mat"] = _matrix(case, wseed)
        s["B"] = _uniform(gen, K, N)
        s["D"] = torch.empty((M, N), dtype=torch.float16, device="cuda")
        if case["beta"] != 0.0:
            s["C"] = _uniform(gen, M, N)
        s["op"] = sb.SpmmBlockwiseOp().initialize(s["mat"], N, s["B"], case["alpha"], s.get("C"), case["beta"], s["D"])
    elif kind == "spmm_host":
        s["mat"] = _matrix(case, wseed)
        s["B"] = _uniform(gen, case["K"], case["N"], pin=True)
        s["D"] = torch.empty((case["M"], case["N"]), dtype=torch.float16).pin_memory()
    elif kind == "linear":
        bias = _uniform(gen, case["M"]) if case["bias"] else None
        s["layer"] = ShflBWLinear(_matrix(case, wseed), bias).cuda()
        s["x"] = _uniform(gen, case["tokens"], case["K"])
    elif kind == "spconv":
        s["filter"] = _filter(case, wseed)
        B, H, W, st = case["B"], case["H"], case["W"], case["stride"]
        s["x"] = _uniform(gen, B, H, W, case["C"])
        s["y"] = torch.empty((B, -(-H // st), -(-W // st), case["F"]), dtype=torch.float16, device="cuda")
        s["op"] = sb.SpconvBlockwiseOp().initialize(s["filter"], B, H, W, st, s["x"], s["y"])
    elif kind == "conv2d":
        bias = _uniform(gen, case["F"]) if case["bias"] else None
        s["layer"] = ShflBWConv2d(_filter(case, wseed), case["stride"], bias).cuda()
        s["x"] = _uniform(gen, case["B"], case["H"], case["W"], case["C"]).permute(0, 3, 1, 2)
    elif kind == "resnet50":
        s["net"] = rn.SparseResNet50(case["B"], hw=case["H"], density=case["density"], V=case["V"], seed=wseed)
        s["net"].x.copy_(_uniform(gen, case["B"], case["H"], case["H"], 64))
        if case["graph"]:
            s["replay"] = s["net"].capture()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "spmm":
        s["op"](torch.cuda.current_stream())
        return s["D"]
    if kind == "spmm_host":
        sb.spmm_host(s["mat"], case["N"], s["B"], s["D"])
        return s["D"]
    if kind in ("linear", "conv2d"):
        return s["layer"](s["x"])
    if kind == "spconv":
        s["op"](torch.cuda.current_stream())
        return s["y"]
    if case["graph"]:
        s["replay"]()
    else:
        s["net"].forward(torch.cuda.current_stream())
    return s["net"].y


# --------------------------------------------------------------------- the same in 64 bits --

def _dense64(m):
    """The dense matrix that a sparse operand's arrays describe, rows in logical order."""
    rows = torch.from_numpy(np.asarray(m.row_permute_ids).copy() if m.row_permute else np.arange(m.nrow)).cuda().long()
    per_block = torch.from_numpy(np.diff(np.asarray(m.indptr)).astype(np.int64)).cuda()
    block = torch.repeat_interleave(torch.arange(len(per_block), device="cuda"), per_block)
    cols = torch.from_numpy(np.asarray(m.indices).astype(np.int64)).cuda()
    values = torch.from_numpy(np.asarray(m.values).view(np.float16).copy()).cuda().double().reshape(-1, m.brow)
    d = torch.zeros((m.nrow, m.ncol), dtype=torch.float64, device="cuda")
    d[rows.reshape(-1, m.brow)[block], cols[:, None]] = values
    return d


def _conv64(x, f, stride):
    """x [B][H][W][C] and a filter whose columns are (r * R + s) * C + c; padding R // 2, outputs ceil(H / stride)."""
    B, H, W, ch = x.shape
    Ho, Wo, R = -(-H // stride), -(-W // stride), f.R
    w = _dense64(f).reshape(f.F, R, R, ch)
    p = torch.nn.functional.pad(x, (0, 0, R // 2, R // 2, R // 2, R // 2))
    out = torch.zeros((B, Ho, Wo, f.F), dtype=torch.float64, device="cuda")
    for r in range(R):
        for c in range(R):
            tap = p[:, r:r + (Ho - 1) * stride + 1:stride, c:c + (Wo - 1) * stride + 1:stride]
            out += tap @ w[:, r, c].t()
    return out


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "spmm":
        y = case["alpha"] * (_dense64(s["mat"]) @ s["B"].double())
        return y + case["beta"] * s["C"].double() if case["beta"] != 0.0 else y
    if kind == "spmm_host":
        return (_dense64(s["mat"]) @ s["B"].cuda().double()).cpu()
    if kind == "linear":
        y = s["x"].double() @ _dense64(s["layer"].spmat).t()
        return y + s["layer"].bias.double() if case["bias"] else y
    if kind == "spconv":
        return _conv64(s["x"].double(), s["filter"], case["stride"])
    if kind == "conv2d":
        y = _conv64(s["x"].permute(0, 2, 3, 1).double(), s["layer"].spfilter, case["stride"])
        return (y + s["layer"].bias.double() if case["bias"] else y).permute(0, 3, 1, 2)
    net = s["net"]
    outs = {-1: net.x.double()}
    last_use = {}
    for i, sp in enumerate(net.specs):
        for j in (sp.src, sp.residual):
            if j is not None:
                last_use[j] = i
    for i, sp in enumerate(net.specs):
        y = net.alphas[i] * _conv64(outs[sp.src], net.filters[i], sp.stride)
        if sp.residual is not None:
            y = y + outs[sp.residual]
        outs[i] = y.clamp_(min=0) if sp.relu else y
        for j in [j for j in outs if last_use.get(j, len(net.specs)) <= i]:
            del outs[j]
    return outs[len(net.specs) - 1]


# -------------------------------------------------------------------------------- cost --

def _sparse_cost(rows, cols, V, density):
    """Non-zero columns over all row blocks, and the bytes of the sparse operand (values, ids, offsets, permutation)."""
    nnzb = rows // V * cols * density
    return nnzb, 2 * nnzb * V + 4 * nnzb + 4 * (rows // V + 1) + 4 * rows


def work(case):
    kind, V, d = case["kind"], case["V"], case["density"]
    if kind in ("spmm", "spmm_host", "linear"):
        M, K = case["M"], case["K"]
        N = case["tokens"] if kind == "linear" else case["N"]
        nnzb, sparse = _sparse_cost(M, K, V, d)
        dense = 2 * K * N + 2 * M * N * (2 if case.get("beta") else 1) + (2 * M if case.get("bias") else 0)
        return {"bytes": sparse + dense, "flops": 2 * nnzb * V * N}
    if kind in ("spconv", "conv2d"):
        B, H, W, Cc, F, R, st = (case[k] for k in ("B", "H", "W", "C", "F", "R", "stride"))
        Ho, Wo = -(-H // st), -(-W // st)
        nnzb, sparse = _sparse_cost(F, R * R * Cc, V, d)
        # a 1x1 filter reads only the pixels that its stride visits
        pixels = Ho * Wo if R == 1 else H * W
        return {"bytes": sparse + 2 * B * (pixels * Cc + Ho * Wo * F) + (2 * F if case.get("bias") else 0),
                "flops": 2 * nnzb * V * B * Ho * Wo}
    # resnet50: layer by layer, every activation written once and read by each layer that takes it
    B, total, flops = case["B"], 0.0, 0.0
    for sp in rn.layer_specs(case["H"]):
        nnzb, sparse = _sparse_cost(sp.F, sp.R * sp.R * sp.C, V, d)
        pixels = sp.Ho * sp.Ho if sp.R == 1 else sp.Hin * sp.Hin
        out = sp.Ho * sp.Ho * sp.F
        total += sparse + 2 * B * (pixels * sp.C + out * (2 if sp.residual is not None else 1))
        flops += 2 * nnzb * V * B * sp.Ho * sp.Ho
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Measured against the same arithmetic with 64-bit sums, times four.  One operator: rounding to
    fp16 is 2.1e-4 of the result's norm, with a bias or beta * C 2.9e-4, and one unit in the last place
    of the largest values 4.4e-3 of the root mean square.  The network rounds after each of 52 layers:
    1.43e-3 and 1.37e-2."""
    if case["kind"] == "resnet50":
        return {"rel": 6e-3, "max": 5.5e-2}
    return {"rel": 1.2e-3, "max": 1.8e-2}
