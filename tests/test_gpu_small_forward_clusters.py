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
    (9, 257, 256, 10, BF16),       # a warp per row
    (9, 257, 256, 10, F32),        # two pieces per lane
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


def test_more_tokens_than_clusters():
    """A key's rows do not fit shared memory, so any token count reads the table in place: past 2^20 tokens a cluster takes several."""
    N, h, r, L = (1 << 20) + 37, 2, 256, 260
    g = torch.Generator(device="cuda").manual_seed(1)
    z = torch.randn(N, h, generator=g, device="cuda")
    C = torch.randn(h, L, r, generator=g, device="cuda") * 0.1
    f = ops.feature_forward(z, C, -3.0, 3.0, L - 2, "relu_sq", 0.75)
    rows = torch.cat([torch.arange(64), torch.randint(0, N, (200,), generator=torch.Generator().manual_seed(2)),
                      torch.arange(N - 100, N)]).cuda()           # the last 37 tokens are second ones of a cluster
    a_ref, d_ref = util.oracle_forward(z[rows], C, -3.0, 3.0, L - 2, "relu_sq", 0.75)
    util.assert_parity("phi(z)", f[rows, :h], a_ref, F32)
    util.assert_parity("lambda*delta", f[rows, h:], d_ref, F32)
    # every row, against calls whose clusters have one token each
    for part in range(0, N, 1 << 19):
        assert torch.equal(f[part:part + (1 << 19)], ops.feature_forward(z[part:part + (1 << 19)], C, -3.0, 3.0, L - 2, "relu_sq", 0.75))
