"""Problems whose operands the tensor-core kernels hold as pairs of f16 (linear spline, h or r that is no multiple of
8 / 16, more than 49 knot rows): float32-accurate results, at the edges of token tiles, key chunks and knot groups."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")

# (N, h, r, G, spline_order)
CASES = [(65, 8, 16, 20, 1), (129, 24, 32, 21, 1), (513, 40, 128, 3, 1), (257, 9, 17, 20, 2), (1000, 101, 20, 12, 2),
         (130, 33, 1, 6, 2), (200, 16, 32, 48, 2), (640, 24, 24, 62, 2), (96, 7, 96, 23, 2),
         (2500, 37, 20, 12, 2)]          # padded rows of dz: more than the blocks that bring them to their place


@pytest.mark.parametrize("case", CASES, ids=lambda c: "N%d_h%d_r%d_G%d_order%d" % c)
def test_split_operands_are_float32_accurate(case):
    N, h, r, G, order = case
    g = torch.Generator().manual_seed(5)
    z = (torch.randn(N, h, generator=g) * 2.0).bfloat16().cuda()
    C = (torch.randn(h, G + order, r, generator=g) * 0.1).bfloat16().cuda()
    go = torch.randn(N, h + r, generator=g).bfloat16().cuda()
    kw = dict(impl="tcgen05", spline_order=order)
    a, d32 = ops.feature_forward(z, C, -3.0, 3.0, G, "gelu", 0.75, delta_f32=True, **kw)
    f = ops.feature_forward(z, C, -3.0, 3.0, G, "gelu", 0.75, **kw)
    dz32, dC, _ = ops.feature_backward(z, C, go, -3.0, 3.0, G, "gelu", 0.75, dz_f32=True, **kw)
    dz, _, dC_cast = ops.feature_backward(z, C, go, -3.0, 3.0, G, "gelu", 0.75, **kw)
    a_ref, d_ref = util.oc.feature_forward(util.f32(z), util.f32(C), -3.0, 3.0, G, "gelu", 0.75, spline_order=order)
    gf = util.f32(go)
    dz_ref, dC_ref = util.oc.feature_backward(util.f32(z), util.f32(C), gf[:, h:], gf[:, :h], -3.0, 3.0, G, "gelu", 0.75,
                                              spline_order=order)
    util.assert_parity("phi(z)", a, a_ref, torch.bfloat16)
    for name, got, ref in (("delta", d32, d_ref), ("dz", dz32, dz_ref), ("dC", dC, dC_ref)):
        util.assert_parity(name, got, ref, torch.float32, rel_gate=2e-5)
    assert torch.equal(f[:, :h], a) and torch.equal(f[:, h:], d32.bfloat16())
    assert torch.equal(dz, dz32.bfloat16()) and torch.equal(dC_cast, dC.bfloat16())
    ops.check_status(z.device)
