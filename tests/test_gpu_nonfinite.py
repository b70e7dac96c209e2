"""Infinities and NaN in C and g_delta reach what touches them and nothing else, on the kernels that promise it: the CUDA-core
family, and the tcgen05 family where it holds operands as pairs of f16 (linear spline, h no multiple of 8, r no multiple
of 16, more than 49 knot rows).  Against the CPU oracle, which adds up the touched rows alone."""
import ctypes

import numpy as np
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")

INF, NAN = float("inf"), float("nan")
# (N, h, r, G, spline_order)
CASES = [(300, 40, 32, 20, 1), (257, 9, 17, 20, 2), (1000, 101, 20, 12, 2), (200, 16, 32, 48, 2), (129, 33, 1, 6, 2),
         (4100, 24, 16, 20, 1)]
IDS = ["N%d_h%d_r%d_G%d_order%d" % c for c in CASES]


def _inputs(N, h, r, G, order, bad, z_std=None):
    gen = torch.Generator().manual_seed(N)
    # inside the grid and below its last interval, where the oracle and the kernels mask alike
    z = (torch.rand(N, h, generator=gen) * 4.8 - 2.8) if z_std is None else torch.randn(N, h, generator=gen) * z_std
    C = torch.randn(h, G + order, r, generator=gen) * 0.1
    go = torch.randn(N, h + r, generator=gen)
    if bad in ("C", "both"):
        C[h // 2, (G + order) // 2, 0] = INF
        C[0, 3, r - 1] = -INF
        C[h - 1, G // 2, r // 2] = NAN
    if bad in ("g", "both"):
        go[N // 3, h] = INF
        go[N - 1, h + r - 1] = NAN
        go[0, h + r // 2] = -INF
    return z.bfloat16().cuda(), C.bfloat16().cuda(), go.bfloat16().cuda()


def _check(name, got, ref, dtype, gate):
    got, ref = util.f32(got), np.asarray(ref, dtype=np.float64)
    fin = np.isfinite(ref)
    assert fin.any()
    extra, missing = np.argwhere(~np.isfinite(got) & fin), np.argwhere(np.isfinite(got) & ~fin)
    assert not len(extra) and not len(missing), f"{name}: {len(extra)} too many, {len(missing)} too few, {extra[:3]} {missing[:3]}"
    util.assert_parity(name, np.where(fin, got, 0.0), np.where(fin, ref, 0.0), dtype, rel_gate=gate)


@pytest.mark.parametrize("impl", ["simt", "tcgen05"])
@pytest.mark.parametrize("bad", ["C", "g", "both"])
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_nonfinite_inputs_stay_where_they_are_touched(case, bad, impl):
    N, h, r, G, order = case
    lo, hi, lam = -3.0, 3.0, 0.75
    z, C, go = _inputs(N, h, r, G, order, bad)
    kw = dict(impl=impl, spline_order=order)
    tc = impl == "tcgen05"
    f = ops.feature_forward(z, C, lo, hi, G, "relu_sq", lam, **kw)
    dz, dC, dC_cast = ops.feature_backward(z, C, go, lo, hi, G, "relu_sq", lam, dz_f32=tc, **kw)
    gf = util.f32(go)
    a_ref, d_ref = util.oc.feature_forward(util.f32(z), util.f32(C), lo, hi, G, "relu_sq", lam, spline_order=order)
    dz_ref, dC_ref = util.oc.feature_backward(util.f32(z), util.f32(C), gf[:, h:], gf[:, :h], lo, hi, G, "relu_sq", lam,
                                              spline_order=order)
    # pairs of f16: 22 bits; bf16 results: half a unit in the eighth bit
    _check("delta", f[:, h:], d_ref, torch.bfloat16, 4e-3)
    _check("dz", dz, dz_ref, torch.float32 if tc else torch.bfloat16, 2e-5 if tc else 4e-3)
    _check("dC", dC, dC_ref, torch.float32, 2e-5)
    _check("dC (bf16)", dC_cast, dC_ref, torch.bfloat16, 4e-3)
    # one result alone, and dz in bf16
    dz1 = ops.feature_backward(z, C, go, lo, hi, G, "relu_sq", lam, need_dC=False, **kw)[0]
    dC1 = ops.feature_backward(z, C, go, lo, hi, G, "relu_sq", lam, need_dz=False, **kw)[1]
    _check("dz alone", dz1, dz_ref, torch.bfloat16, 4e-3)
    _check("dC alone", dC1, dC_ref, torch.float32, 2e-5)
    ops.check_status(z.device)


@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_nonfinite_inputs_and_tokens_outside_the_grid(case):
    N, h, r, G, order = case
    z, C, go = _inputs(N, h, r, G, order, "both", z_std=2.5)
    got = {}
    for impl in ("simt", "tcgen05"):
        f = ops.feature_forward(z, C, -3.0, 3.0, G, "gelu", 0.5, impl=impl, spline_order=order)
        dz, dC, _ = ops.feature_backward(z, C, go, -3.0, 3.0, G, "gelu", 0.5, impl=impl, spline_order=order)
        got[impl] = f, dz, dC
    for name, a, b in zip(("f", "dz", "dC"), got["tcgen05"], got["simt"]):
        _check(name, a, util.f32(b), torch.bfloat16, 1e-2)


# (N, h, r, lanes that add up the splits of an output): more than 16, 32 and 64 key splits
@pytest.mark.parametrize("N,h,r,lanes", [(320, 640, 32, 2), (319, 2560, 32, 4), (320, 5120, 16, 8)])
@pytest.mark.parametrize("delta_f32", [False, True])
def test_nonfinite_code_tables_and_many_key_splits(N, h, r, lanes, delta_f32):
    z, C, _ = _inputs(N, h, r, 20, 1, "C")
    p = ops._problem(z, C, -3.0, 3.0, 20, "relu_sq", 0.75, "tcgen05", 1)
    image = 4096 + -(-h * 24 * r * 2 // 256) * 256       # header and operand image of C: what is left of the scratch are the partials
    partials = ops._lib.load().skv_scratch_bytes(ctypes.byref(p), ops._lib.SKV_OP_FORWARD) - image
    assert partials // (N * r * 4) > 8 * lanes
    f = ops.feature_forward(z, C, -3.0, 3.0, 20, "relu_sq", 0.75, impl="tcgen05", spline_order=1, delta_f32=delta_f32)
    _, d_ref = util.oc.feature_forward(util.f32(z), util.f32(C), -3.0, 3.0, 20, "relu_sq", 0.75, spline_order=1)
    # float32: pairs of f16 and sums of a few thousand products; bf16: half a unit in the eighth bit
    if delta_f32:
        _check("delta", f[1], d_ref, torch.float32, 2e-5)
    else:
        _check("delta", f[:, h:], d_ref, torch.bfloat16, 4e-3)
    ops.check_status(z.device)
