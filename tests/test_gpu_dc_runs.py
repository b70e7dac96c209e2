"""dC at the edges of its plan, with scratch that holds NaN beforehand, against the CPU oracle: slabs that are a whole number
of runs, more than 32 runs in a slab, fewer than four slabs, runs that cross slabs, runs longer than a slab."""
import ctypes

import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

_lib = pytest.importorskip("sparsespline_ffn_b200._lib")

# (N, h, L, r, spline_order, does a run cross slabs, runs per slab or 0 for a run longer than a slab)
CASES = [(94720, 32, 22, 128, 2, False, 74), (513856, 256, 22, 32, 2, False, 37), (103461, 8, 42, 16, 2, False, 147),
         (58151, 8, 41, 16, 1, True, 130), (2325, 2496, 42, 32, 2, True, 2), (1828, 4760, 42, 32, 2, True, 0)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "N%d_h%d_L%d_r%d_order%d" % c[:5])
def test_dc_adds_what_was_written(case):
    N, h, L, r, order, crosses, runs = case
    lo, hi, G, lam = -3.0, 3.0, L - order, 0.75
    lib = _lib.load()
    g = torch.Generator().manual_seed(9)
    z = (torch.randn(N, h, generator=g) * 1.5).bfloat16()
    go = torch.randn(N, r, generator=g).bfloat16()
    C = torch.zeros(h, L, r, dtype=torch.bfloat16)
    zd, gd, Cd = z.cuda(), go.cuda(), C.cuda()
    p = _lib.Problem(N=N, h=h, L=L, r=r, grid_lo=lo, scale=G / (hi - lo), lambda_scale=lam, activation=0, dtype=0, impl=2,
                     spline_order=order)
    plan = (ctypes.c_int64 * 8)()
    _lib.check(lib.skv_debug_dc_plan(ctypes.byref(p), 0, plan))
    assert bool(plan[0]) == crosses and (plan[3] > plan[1] if runs == 0 else plan[7] == runs), list(plan)
    need = int(lib.skv_scratch_bytes(ctypes.byref(p), _lib.SKV_OP_BACKWARD))
    scratch = torch.full((need // 4 + 1,), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    dC = torch.full((h, L, r), float("nan"), device="cuda")
    _lib.check(lib.skv_feature_backward(
        ctypes.byref(p), zd.data_ptr(), h, Cd.data_ptr(), None, 0, gd.data_ptr(), r, None, h, dC.data_ptr(), None,
        scratch.data_ptr(), need, status.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    _, ref = util.oc.feature_backward(util.f32(z), util.f32(C), util.f32(go), None, lo, hi, G, "identity", lam,
                                      spline_order=order)
    # f16 operands (a weight rounded to 11 bits), or pairs of them for the linear spline; float32 sums
    util.assert_parity("dC", dC, ref, torch.bfloat16, rel_gate=2e-3 if order == 2 else 2e-5)
