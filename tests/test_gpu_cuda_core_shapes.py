"""The CUDA-core kernels at the edges of their tiles: tokens around a lane group, a warp and a tile, keys around a slab and the warps of a
CTA, rows that are read in pieces of 16 bytes, of 4 elements or one by one, wide rows, many intervals, a key's accumulator that does not
fit shared memory; against the CPU oracle."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")

F32, BF16 = torch.float32, torch.bfloat16


@pytest.mark.parametrize("N,h,r,L,order,dtype", [
    (1, 1, 4, 4, 2, F32),
    (65, 23, 32, 22, 2, F32),
    (255, 24, 32, 22, 2, F32),
    (257, 25, 32, 21, 1, F32),
    (513, 49, 64, 22, 2, F32),
    (300, 65, 33, 10, 2, F32),     # channels one by one
    (130, 33, 20, 42, 2, F32),     # a lane group that is not full
    (129, 31, 8, 22, 2, F32),
    (200, 40, 128, 22, 2, F32),    # transposes of eight keys by 32 lanes
    (200, 40, 16, 101, 2, F32),    # more intervals than lanes
    (190, 27, 200, 22, 2, F32),    # two pieces per lane
    (190, 27, 200, 22, 2, BF16),
    (140, 19, 256, 22, 2, BF16),
    (600, 37, 136, 22, 2, BF16),   # wide bf16 rows staged (more tokens than are read in place), a ragged last slab
    (1025, 19, 200, 22, 2, BF16),
    (577, 45, 256, 21, 1, BF16),
    (90, 3, 256, 700, 2, F32),     # a key's rows and accumulator do not fit shared memory
])
def test_cuda_core_kernels(N, h, r, L, order, dtype):
    G, lo, hi, lam = L - order, -3.0, 3.0, 0.75
    z = util.make_inputs(N, h, r, 2, dtype, z_scale=1.5)[0]
    C = (torch.randn(h, L, r, generator=torch.Generator().manual_seed(3)) * 0.1).to(dtype).cuda()
    go = torch.randn(N, h + r, generator=torch.Generator().manual_seed(4)).to(dtype).cuda()
    kw = dict(impl="simt", spline_order=order)
    f = ops.feature_forward(z, C, lo, hi, G, "gelu", lam, **kw)
    dz, dC, _ = ops.feature_backward(z, C, go, lo, hi, G, "gelu", lam, **kw)
    dz0 = ops.feature_backward(z, C, go[:, h:].contiguous(), lo, hi, G, "gelu", lam, with_base=False, **kw)[0]
    dC1 = ops.feature_backward(z, C, go, lo, hi, G, "gelu", lam, need_dz=False, **kw)[1]
    gf = util.f32(go)
    a_ref, d_ref = util.oc.feature_forward(util.f32(z), util.f32(C), lo, hi, G, "gelu", lam, spline_order=order)
    dz_ref, dC_ref = util.oc.feature_backward(util.f32(z), util.f32(C), gf[:, h:], gf[:, :h], lo, hi, G, "gelu", lam, spline_order=order)
    dz0_ref, _ = util.oc.feature_backward(util.f32(z), util.f32(C), gf[:, h:], None, lo, hi, G, "gelu", lam, spline_order=order)
    # float32: sums of up to a thousand products; the base path's erf and exp differ in their last bits
    gate = 1e-5 if dtype == F32 else None
    for name, got, ref in (("phi(z)", f[:, :h], a_ref), ("delta", f[:, h:], d_ref), ("dz", dz, dz_ref), ("dz of the spline", dz0, dz0_ref)):
        util.assert_parity(name, got, ref, dtype, rel_gate=gate)
    util.assert_parity("dC", dC, dC_ref, F32, rel_gate=1e-5)
    assert torch.equal(dC, dC1)                       # dC as the first kernel of a call, and beside dz
