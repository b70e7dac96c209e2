"""The forward of few tokens, a cluster of CTAs per token: cluster sizes, ragged shares of keys, rows that cannot be read in
16-byte pieces, a key's table larger than shared memory."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")

BF16, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("N,h,r,L,dtype", [
    (1, 1, 16, 22, BF16),          # fewer keys than CTAs of a cluster
    (2, 5119, 32, 22, BF16),       # a ragged last share
    (17, 5120, 32, 22, BF16),      # eight CTAs per token, more than one wave of clusters of the largest CTAs
    (120, 640, 32, 22, BF16),
    (500, 63, 64, 22, BF16),       # one CTA per token
    (3, 300, 33, 14, BF16),        # channels one by one
    (9, 257, 256, 10, BF16),       # two pieces per lane
    (64, 1536, 64, 22, F32),
    (5, 100, 7, 8, F32),
    (70, 5, 256, 1000, F32),       # no room for a key's rows: any token count
])
def test_small_forward_clusters(N, h, r, L, dtype):
    z, C, _ = util.make_inputs(N, h, r, L - 2, dtype)
    f = ops.feature_forward(z, C, -3.0, 3.0, L - 2, "relu_sq", 0.75)
    a_ref, d_ref = util.oracle_forward(z, C, -3.0, 3.0, L - 2, "relu_sq", 0.75)
    util.assert_parity("phi(z)", f[:, :h], a_ref, dtype)
    util.assert_parity("lambda*delta", f[:, h:], d_ref, dtype)
    ops.check_status(z.device)
