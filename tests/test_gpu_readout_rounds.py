"""The read-out GEMM where whole rounds of tiles are followed by K slices of the remaining ones (both tile heights, ragged tokens and
outputs), against a float64 product of the feature."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")


@pytest.mark.parametrize("act", ["relu_sq", "identity"])
@pytest.mark.parametrize("shape", [(2500, 2048, 32, 2040), (8192, 2560, 16, 1280), (2560, 2056, 64, 2048)],
                         ids=lambda s: "N%d_h%d_r%d_D%d" % s)
def test_rounds_and_slices(shape, act):
    N, h, r, D = shape
    z, C, _ = util.make_inputs(N, h, r, 20, torch.bfloat16)
    W = (torch.randn(D, h + r, generator=torch.Generator().manual_seed(2)) * 0.05).bfloat16().cuda()
    f = ops.feature_forward(z, C, -3.0, 3.0, 20, act, 0.5)
    y = ops.feature_readout_forward(z, C, W, -3.0, 3.0, 20, act, 0.5)
    ref = (f.double() @ W.double().T).float().cpu().numpy()
    util.assert_parity("y", y, ref, torch.bfloat16, rel_gate=5e-3)
    assert torch.equal(y, ops.feature_readout_forward(z, C, W, -3.0, 3.0, 20, act, 0.5))
    ops.check_status(z.device)
