"""The read-out GEMM where whole rounds of tiles are followed by K slices of the remaining ones (both tile heights, either activation,
ragged tokens and outputs), and where all tiles are whole, against a float64 product of the feature."""
import ctypes

import pytest
import torch

from sparsespline_ffn_b200 import _lib
from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")


def _check(shape, act):
    N, h, r, D = shape
    z, C, _ = util.make_inputs(N, h, r, 20, torch.bfloat16)
    W = (torch.randn(D, h + r, generator=torch.Generator().manual_seed(2)) * 0.05).bfloat16().cuda()
    f = ops.feature_forward(z, C, -3.0, 3.0, 20, act, 0.5)
    y = ops.feature_readout_forward(z, C, W, -3.0, 3.0, 20, act, 0.5)
    ref = (f.double() @ W.double().T).float().cpu().numpy()
    util.assert_parity("y", y, ref, torch.bfloat16, rel_gate=5e-3)
    assert torch.equal(y, ops.feature_readout_forward(z, C, W, -3.0, 3.0, 20, act, 0.5))
    ops.check_status(z.device)


def _plan(shape, act):
    N, h, r, D = shape
    p = _lib.Problem(N=N, h=h, L=22, r=r, grid_lo=-3.0, scale=20.0 / 6.0, lambda_scale=0.5, activation=_lib.SKV_ACT[act],
                     dtype=_lib.SKV_BF16, impl=_lib.SKV_IMPL["auto"], spline_order=2)
    out = (ctypes.c_int64 * 4)()
    _lib.check(_lib.load().skv_debug_readout_plan(ctypes.byref(p), D, out))
    return dict(zip(("tokens", "tiles", "whole", "slices"), out))


# (shape, activation, tokens of a tile, whole rounds).  The last tile of tokens is ragged but at 8192, the last of outputs at 2040 and 1016.
MIXED = [((2500, 2560, 32, 2040), "relu_sq", 128, 1), ((9473, 2048, 64, 1016), "identity", 128, 2),
         ((8192, 5120, 32, 1280), "relu_sq", 128, 2), ((8192, 5120, 32, 1280), "identity", 128, 2),
         ((4737, 4104, 32, 2040), "relu_sq", 256, 1), ((9601, 6144, 16, 2040), "identity", 256, 2)]
IDS = [f"N{s[0]}_h{s[1]}_r{s[2]}_D{s[3]}-{a}" for s, a, *_ in MIXED]


@pytest.mark.parametrize("shape,act,tokens,rounds", MIXED, ids=IDS)
def test_rounds_then_slices(shape, act, tokens, rounds):
    plan = _plan(shape, act)
    assert plan["tokens"] == tokens and plan["whole"] == 148 * rounds < plan["tiles"] and plan["slices"] > 1, plan
    _check(shape, act)


@pytest.mark.parametrize("act", ["relu_sq", "identity"])
@pytest.mark.parametrize("shape", [(2500, 2048, 32, 2040), (8192, 2560, 16, 1280), (2560, 2056, 64, 2048)],
                         ids=lambda s: "N%d_h%d_r%d_D%d" % s)
def test_rounds_and_slices(shape, act):
    _check(shape, act)
