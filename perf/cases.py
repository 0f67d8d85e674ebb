"""Performance cases of the INT8 linear library: what its users run, through the public entry points.

A case names an entry point ("op"), its sizes and its options:
  infer      Int8Linear forward without gradients (serving: prefill and small batches of tokens)
  train      Int8Linear forward + backward (Y, dX, dW, bias gradient) through autograd
  block_fwd  block_channel.fwd_32   a [B, M, K] x b [N, K]
  block_bwd  block_channel.bwd_33   a [B, M, K] x b [B, N, K]
  dc_fwd     double_channel.fwd_32  a [B, M, K] x b [N, K]
  dc_bwd     double_channel.bwd_33  a [B, M, K] x b [B, N, K]
  fused_fwd  fused.fwd_32           a [B, M, K] x b [N, K]
  fused_bwd  fused.bwd_33           a [B, M, K] x b [B, N, K]

Sizes follow the library's own configurations (the 512x1024x1024 linear, the double_channel forward at
8192x4096x4096, the Llama-2-7B and Llama-70B MLP shapes, the 8192^3 square) and odd multiples of 128, the
granularity that every entry point asks for.  Data follow them too: activations ~ N(0,1) with 0.5 % outlier
channels x30, weights ~ N(0,0.02), output gradients ~ N(0,1e-3), bias ~ N(0,0.01), all bf16.

The linears of a decoder layer stand here one by one.  Chained, a single flipped bf16 rounding moves int8
roundings of the next layer and two correct runs drift apart by the quantization noise itself (2e-2 to 5e-2
after seven linears, measured), which says nothing about either of them.
"""
import math

import torch

from triton_int8_b200 import block_channel, double_channel, fused
from triton_int8_b200.linear import Int8Config, Int8Linear

_LARGEST = dict(M=32768, K=8192, N=28672)


def listed():
    return [
        # The smallest call in earnest: one 128-token block through a small serving layer.
        dict(name="infer 128x1024x1024", op="infer", M=128, K=1024, N=1024, bias=True, scaling="tile128", round="half_up", hadamard=0),
        # Short prompt through a 7B up-projection: the weight, not the tokens, is the work.
        dict(name="infer 256x4096x11008", op="infer", M=256, K=4096, N=11008, bias=False, scaling="tile128", round="half_up", hadamard=128),
        # One training step of the smallest configured linear, where launches and host work count.
        dict(name="train 512x1024x1024", op="train", M=512, K=1024, N=1024, bias=True, scaling="tile128", round="half_up", hadamard=0),
        # The finer per-(row,128) grouping with round-to-nearest-even, at sizes that fill no tile grid evenly.
        dict(name="train row128 1920x1408x2176", op="train", M=1920, K=1408, N=2176, bias=True, scaling="row128", round="rne", hadamard=0),
        # Per-row scaling over the whole contraction for all three products of a mid-size layer.
        dict(name="train dc 4096x4096x4096", op="train", M=4096, K=4096, N=4096, bias=True, scaling="double_channel", round="half_up", hadamard=0),
        # Rotated training step of the Llama-2-7B up-projection.
        dict(name="train rot 16384x4096x11008", op="train", M=16384, K=4096, N=11008, bias=False, scaling="tile128", round="half_up", hadamard=128),
        # Rotated training step of the Llama-70B MLP layer: the benchmark's shape and the largest case.
        dict(name="train rot 32768x8192x28672", op="train", bias=False, scaling="tile128", round="half_up", hadamard=128, **_LARGEST),
        # Training step of the Llama-2-7B down-projection at the token count of the decoder-layer workload.
        dict(name="train 8192x11008x4096", op="train", M=8192, K=11008, N=4096, bias=False, scaling="tile128", round="half_up", hadamard=0),
        # Operator-level forward with the whole-row rotation and a bias.
        dict(name="dc_fwd 8192x4096x4096", op="dc_fwd", B=1, M=8192, K=4096, N=4096, bias=True, hadamard="full"),
        # The square block-scaled forward on which the GEMM is judged.
        dict(name="block_fwd 8192x8192x8192", op="block_fwd", B=1, M=8192, K=8192, N=8192, bias=False, scaling="tile128", hadamard=0),
        # Batched product of two activations-like operands at ragged sizes.
        dict(name="block_bwd 3x640x1920x896", op="block_bwd", B=3, M=640, K=1920, N=896, scaling="tile128", hadamard=0),
        # The fused variant's forward, batched.
        dict(name="fused_fwd 2x1024x2048x1536", op="fused_fwd", B=2, M=1024, K=2048, N=1536),
    ]


def _spread(rng, lo, hi, step=128):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["infer", "infer", "train", "train", "train", "train", "block_fwd", "block_bwd", "dc_fwd",
                     "dc_bwd", "fused_fwd", "fused_bwd"])
    while True:
        M, K, N = _spread(rng, 128, 32768), _spread(rng, 256, 11008), _spread(rng, 256, 28672)
        B = 1 if op in ("infer", "train") else rng.choice([1, 1, 2, 3, 4])
        case = dict(op=op, M=M, K=K, N=N)
        if op in ("infer", "train"):
            case.update(bias=rng.random() < 0.5, scaling=rng.choice(["tile128", "tile128", "tile128", "row128", "double_channel"]),
                        hadamard=rng.choice([0, 128]))
            case["round"] = "rne" if case["scaling"] == "row128" else "half_up"
        else:
            case["B"] = B
            if op == "block_fwd":
                case.update(bias=rng.random() < 0.5, scaling=rng.choice(["tile128", "tile128", "row128"]), hadamard=rng.choice([0, 128]))
            elif op == "block_bwd":
                case.update(scaling="tile128", hadamard=rng.choice([0, 128]))
            elif op in ("dc_fwd", "dc_bwd"):
                case["hadamard"] = rng.choice(["full", "none"])
                if case["hadamard"] == "full":   # the whole-row rotation is defined for powers of two
                    case["K"] = 1 << rng.randint(8, 13)
                if op == "dc_fwd":
                    case["bias"] = rng.random() < 0.5
        products = 3 if op == "train" else 1
        if B * M * case["K"] * N * products <= 3 * math.prod(_LARGEST.values()) and B * M * N <= _LARGEST["M"] * _LARGEST["N"]:
            return case


# ------------------------------------------------------------------------------------------------ inputs
def _normal(g, shape, std, dev="cuda"):
    return torch.empty(shape, dtype=torch.bfloat16, device=dev).normal_(0.0, std, generator=g)


def _activations(g, shape):
    """~ N(0,1) with 0.5 % of the channels (last axis) x30."""
    x = _normal(g, shape, 1.0)
    n_out = -(-shape[-1] * 5 // 1000)
    x[..., torch.randperm(shape[-1], generator=g, device="cuda")[:n_out]] *= 30
    return x


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    M, K, N = case["M"], case["K"], case["N"]
    if op in ("infer", "train"):
        lin = Int8Linear(K, N, bias=case["bias"], device="cuda",
                         config=Int8Config(scaling=case["scaling"], round=case["round"], hadamard=case["hadamard"]))
        with torch.no_grad():
            lin.weight.normal_(0.0, 0.02, generator=g)
            if case["bias"]:
                lin.bias.normal_(0.0, 0.01, generator=g)
        state = dict(op=op, lin=lin, x=_activations(g, (M, K)))
        if op == "train":
            state["x"].requires_grad_(True)
            state["dy"] = _normal(g, (M, N), 1e-3)
        return state
    B = case["B"]
    a = _activations(g, (B, M, K))
    if op.endswith("_fwd"):
        b = _normal(g, (N, K), 0.02)
    else:
        b = _normal(g, (B, N, K), 1.0)
    kw = {}
    if case.get("bias"):
        kw["bias"] = _normal(g, (N,), 0.01)
    if op.startswith("block"):
        kw.update(scaling=case["scaling"], hadamard=case["hadamard"])
        if case["scaling"] == "row128":
            kw["round"] = "rne"
    elif op.startswith("dc"):
        kw["hadamard"] = case["hadamard"]
    return dict(op=op, a=a, b=b, kw=kw)


_CALLS = {
    "block_fwd": block_channel.fwd_32, "block_bwd": block_channel.bwd_33,
    "dc_fwd": double_channel.fwd_32, "dc_bwd": double_channel.bwd_33,
    "fused_fwd": fused.fwd_32, "fused_bwd": fused.bwd_33,
}


def run(state):
    op = state["op"]
    if op == "infer":
        with torch.no_grad():
            return state["lin"](state["x"])
    if op == "train":
        lin, x = state["lin"], state["x"]
        y = lin(x)
        y.backward(state["dy"])
        out = {"y": y.detach(), "dx": x.grad}
        for name, p in lin.named_parameters():
            out["d " + name] = p.grad
            p.grad = None
        x.grad = None
        return out
    return _CALLS[op](state["a"], state["b"], **state["kw"])


# ------------------------------------------------------------------------------------------------ work
def work(case):
    op = case["op"]
    M, K, N, B = case["M"], case["K"], case["N"], case.get("B", 1)
    bias = N if case.get("bias") else 0
    if op == "train":   # x, w, bias, dy in; y, dx, dw, dbias out
        return {"bytes": 2 * (2 * M * K + 2 * N * K + 2 * M * N + 2 * bias), "flops": 3 * 2 * M * K * N}
    b_batch = B if op.endswith("_bwd") else 1
    return {"bytes": 2 * (B * M * K + b_batch * N * K + B * M * N + bias), "flops": 2 * B * M * K * N}


def tolerance(case):
    # Integers and scales are fixed.  What another correct implementation may do differently is the order of
    # the fp32 operations in front of the bf16 rounding, which flips single roundings (one unit in the last
    # place of a bf16 is at most 7.8e-3 of the value).  Measured between the two operation orders that the
    # library has: up to 8.1e-4 for the sums over K blocks, 2e-5 for the two scalings of whole-K products.
    whole_k = case["op"].startswith("dc") or case.get("scaling") == "double_channel"
    return {"rel": 1e-4 if whole_k else 3e-3, "max": 0.03}
