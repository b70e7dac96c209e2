"""The read-out GEMM's tile heights and K slices (few tokens, several waves, ragged tiles) against a float64 product of the
feature."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")


@pytest.mark.parametrize("act", ["relu_sq", "identity"])
@pytest.mark.parametrize("shape", [(1, 512, 32, 264), (129, 1288, 64, 256), (700, 64, 16, 8), (4100, 328, 32, 1280)],
                         ids=lambda s: "N%d_h%d_r%d_D%d" % s)
def test_readout_matches_the_product_of_the_feature(shape, act):
    N, h, r, D = shape
    z, C, _ = util.make_inputs(N, h, r, 20, torch.bfloat16)
    W = (torch.randn(D, h + r, generator=torch.Generator().manual_seed(2)) * 0.05).bfloat16().cuda()
    f = ops.feature_forward(z, C, -3.0, 3.0, 20, act, 0.5)
    y = ops.feature_readout_forward(z, C, W, -3.0, 3.0, 20, act, 0.5)
    ref = (f.double() @ W.double().T).float().cpu().numpy()
    util.assert_parity("y", y, ref, torch.bfloat16, rel_gate=5e-3)
    assert torch.equal(y, ops.feature_readout_forward(z, C, W, -3.0, 3.0, 20, act, 0.5))
    ops.check_status(z.device)
