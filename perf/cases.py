"""The calls whose speed matters to users of this package, as measurable cases.

Each case is one pass through the public operators as a user's program makes it: a training step of the
feature operator (forward, then backward through autograd), an inference forward, the delta-only operator,
the fused read-out and the linear spline.  Sizes are the benchmark's configurations (h = 5120 keys, G = 20,
r = 32, the rank/grid sweep, the float32 layer of N = 4096, h = 1024), the layer's defaults (r = 64, grid
[-3, 3]) and ordinary sizes in between, ragged ones among them.  ``draw`` spreads over the same ranges.
"""
import math

import torch

from sparsespline_ffn_b200 import flash_spline_delta, flash_spline_feature
from sparsespline_ffn_b200.cuda_ext import spline_kv_fwd_fused_cuda

_DTYPE = {"bf16": torch.bfloat16, "f32": torch.float32}


def _case(op, N, h, r=32, G=20, dtype="bf16", act="relu_sq", order=2, grid=5.0, lam=1.0, z_std=1.0, d_out=0):
    return dict(op=op, N=N, h=h, r=r, G=G, dtype=dtype, act=act, order=order, grid=grid, lam=lam, z_std=z_std,
                d_out=d_out)


def listed():
    cases = {
        # one decoding step of a small batch of sequences at the d20 width: latency and launches
        "decode_16": _case("infer", 16, 5120),
        # a prompt of odd length at the reference's production width
        "prefill_1999": _case("infer", 1999, 2560),
        # inference through the layer's fused read-out, d_out = the model width
        "readout_8k": _case("readout", 8192, 5120, d_out=1280),
        # the headline: one training step of one d20 layer
        "train_d20": _case("train", 65536, 5120),
        # the boundary-heavy d20 configuration (lambda warm-up, wide pre-activations) at a micro-batch
        "train_wide_8k": _case("train", 8192, 5120, lam=0.25, z_std=2.0),
        # the layer's default rank and grid at a small model's width, a ragged micro-batch, gelu base path
        "train_small_gelu": _case("train", 3001, 768, r=64, act="gelu", grid=3.0),
        # the rank and grid ends of the sweep
        "train_r128": _case("train", 65536, 5120, r=128),
        "train_g40": _case("train", 16384, 5120, G=40),
        # the residual-only operator (layers without a base path)
        "delta_r64": _case("delta", 8192, 2560, r=64, grid=3.0),
        # the float32 layer configuration
        "train_f32": _case("train", 4096, 1024, dtype="f32"),
        # the linear spline under bf16
        "train_linear": _case("train", 4096, 1024, order=1),
        # a width and a rank that are no multiples of anything
        "train_odd": _case("train", 2000, 1001, r=20, G=12, grid=3.0),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    """Log-uniform integer; half the time rounded to two binary digits, otherwise left odd."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 0.5:
        step = 1 << max(0, int(math.log2(v)) - 1)
        return int(max(lo, min(hi, round(v / step) * step)))
    return int(max(lo, min(hi, int(v) | 1)))


def draw(rng):
    kind = rng.choice(["infer", "infer", "train", "train", "train", "delta", "readout", "f32", "linear", "odd"])
    grid = rng.choice([3.0, 5.0])
    act = rng.choice(["relu_sq", "relu_sq", "identity", "gelu"])
    lam, z_std = rng.choice([0.25, 0.5, 1.0]), rng.choice([1.0, 1.0, 1.5, 2.0])
    h = 8 * _log_int(rng, 48, 640)
    r = rng.choice([16, 32, 32, 64, 128])
    G = rng.choice([20, 20, 20, 8, 14, 30, 40]) if r < 128 else 20      # the sweep moves rank or grid, not both
    if kind == "infer":
        return _case("infer", _log_int(rng, 1, 16384), h, r, G, act=act, grid=grid, lam=lam, z_std=z_std)
    if kind == "train":
        return _case("train", _log_int(rng, 256, 32768), h, r, G, act=act, grid=grid, lam=lam, z_std=z_std)
    if kind == "delta":
        return _case("delta", _log_int(rng, 256, 32768), h, r, G, grid=grid, lam=lam, z_std=z_std)
    if kind == "readout":
        return _case("readout", _log_int(rng, 16, 16384), h, r, G, act=rng.choice(["relu_sq", "identity"]), grid=grid,
                     lam=lam, z_std=z_std, d_out=8 * _log_int(rng, 32, 256))
    if kind == "f32":
        return _case(rng.choice(["train", "train", "infer"]), _log_int(rng, 64, 4096), _log_int(rng, 128, 1536),
                     rng.choice([16, 32, 32, 64]), G, "f32", act, grid=grid, lam=lam, z_std=z_std)
    if kind == "linear":
        return _case("train", _log_int(rng, 128, 4096), 8 * _log_int(rng, 16, 192), rng.choice([16, 32, 64]), G,
                     rng.choice(["bf16", "bf16", "f32"]), act, order=1, grid=grid, lam=lam, z_std=z_std)
    return _case(rng.choice(["train", "train", "infer"]), _log_int(rng, 64, 4096), _log_int(rng, 128, 1536),
                 rng.choice([8, 12, 20, 24, 33, 40]), G, "bf16", act, grid=grid, lam=lam, z_std=z_std)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _DTYPE[case["dtype"]]
    N, h, r = case["N"], case["h"], case["r"]
    train = case["op"] in ("train", "delta")

    def normal(*shape, std=1.0):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype).mul_(std)

    st = {"case": case, "z": normal(N, h, std=case["z_std"]).requires_grad_(train),
          "C": normal(h, case["G"] + case["order"], r, std=0.02).requires_grad_(train)}
    if train:
        st["go"] = normal(N, r if case["op"] == "delta" else h + r)
    if case["op"] == "readout":
        st["W"] = normal(case["d_out"], h + r, std=(h + r) ** -0.5)
    return st


def run(state):
    c, z, C = state["case"], state["z"], state["C"]
    lo, hi, G, lam = -c["grid"], c["grid"], c["G"], c["lam"]
    if c["op"] == "readout":
        return spline_kv_fwd_fused_cuda(z, C, state["W"], lo, hi, G, c["act"], lam)
    if c["op"] == "infer":
        with torch.no_grad():
            return flash_spline_feature(z, C, lo, hi, G, c["act"], lam)
    z.grad = C.grad = None
    if c["op"] == "delta":
        f = flash_spline_delta(z, C, lo, hi, G, lam)
    else:
        f = flash_spline_feature(z, C, lo, hi, G, c["act"], lam, spline_order=c["order"])
    f.backward(state["go"])
    return f, z.grad, C.grad


def work(case):
    """Inputs once, outputs once; per (token, key) pair one multiply-add per code channel for each of the
    order + 1 knot rows a value touches (forward, dC and dz each), and the read-out product."""
    N, h, r, L = case["N"], case["h"], case["r"], case["G"] + case["order"]
    rows = case["order"] + 1
    size = 4 if case["dtype"] == "f32" else 2
    table = min(L, rows * N) * h * r * size
    width = r if case["op"] == "delta" else h + r
    if case["op"] == "readout":
        D = case["d_out"]
        return {"bytes": size * (N * h + D * (h + r) + N * D) + table,
                "flops": 2 * rows * N * h * r + 2 * N * D * (h + r)}
    nbytes = size * (N * h + N * width) + table
    flops = 2 * rows * N * h * r
    if case["op"] != "infer":
        nbytes += size * (2 * N * h + N * width) + table + size * h * L * r
        flops *= 3
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # float32: sums of up to a few thousand rounded products; bf16: results rounded to 8 bits
    return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-2}
