"""Forwards on both sides of the token count up to which table rows are gathered in place, against the CPU oracle."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")


@pytest.mark.parametrize("N,h,r,G", [(1, 8, 16, 20), (3, 520, 20, 12), (88, 2600, 32, 20), (133, 5120, 32, 20),
                                     (512, 72, 128, 20), (513, 72, 128, 20)])
def test_small_forward_matches_the_oracle(N, h, r, G):
    z, C, _ = util.make_inputs(N, h, r, G, torch.bfloat16)
    f = ops.feature_forward(z, C, -3.0, 3.0, G, "relu_sq", 0.75)
    a_ref, d_ref = util.oracle_forward(z, C, -3.0, 3.0, G, "relu_sq", 0.75)
    util.assert_parity("phi(z)", f[:, :h], a_ref, torch.bfloat16)
    util.assert_parity("lambda*delta", f[:, h:], d_ref, torch.bfloat16)
    ops.check_status(z.device)
