"""Long sums of the tcgen05 kernels.  The tensor core cuts an accumulator off towards zero at every MMA, an error that grows
with their number and never averages out, so an accumulator takes a bounded number of them.  All summands are
positive here, so that every bit lost counts; the oracle gets a few keys (dC) and a few tokens (delta), which depend on
nothing else."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")

LO, HI = -5.0, 5.0


def _normal(*shape, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.bfloat16)


def _dC_of(z, C, g, G, order, keys):
    return util.oc.feature_backward(util.f32(z[:, keys]), util.f32(C[keys]), util.f32(g), None, LO, HI, G, "identity", 1.0,
                                    spline_order=order)[1]


@pytest.mark.parametrize("N,h,r", [(65536, 11840, 32), (40000, 2368, 128)])
def test_dC_of_many_tokens_per_accumulator(N, h, r):
    # pre-activations that are multiples of 1/8 have weights that are multiples of 1/32: the f16 operands are exact, and
    # the float32 sums are all that is left.  192 tiles x 4 MMAs, each at most 2^-23 of the sum so far (half of it on
    # the average, and the sum grows): below 768 x 2^-24 x 1/2 = 2.3e-5
    G = 20
    z = (_normal(N, h, seed=1) * 8).round() / 8
    g = _normal(N, r, seed=2).abs()
    C = torch.zeros(h, G + 2, r, dtype=torch.bfloat16, device="cuda")
    _, dC, _ = ops.feature_backward(z, C, g, LO, HI, G, "identity", 1.0, with_base=False, need_dz=False, cast_dC=False,
                                    impl="tcgen05")
    for keys in (slice(0, 4), slice(h - 4, h)):
        util.assert_parity("dC", dC[keys], _dC_of(z, C, g, G, 2, keys), torch.bfloat16, bias=True, rel_gate=2.3e-5)
    ops.check_status(z.device)


@pytest.mark.parametrize("N,h,r,G,order", [(20000, 5113, 32, 20, 2), (33000, 4096, 32, 20, 1), (2000, 1001, 20, 12, 2),
                                           (9000, 1536, 33, 20, 2), (600, 8 * 8 * 16 + 1, 20, 48, 2)])
def test_pairs_of_f16_keep_their_accuracy(N, h, r, G, order):
    # forward: 8 chunks of 8 keys, dC: 16 tiles of 64 tokens to an accumulator, 64 to 256 MMAs, each at most 2^-23 of
    # the sum so far, 2^-24 of the final one on the average: 128 x 2^-24 x 1/2 = 4e-6 for dC, and 22 bits of the operands
    z, g = _normal(N, h, seed=1), _normal(N, r, seed=2).abs()
    C = (_normal(h, G + order, r, seed=3) * 0.02).abs()
    kw = dict(impl="tcgen05", spline_order=order, with_base=False)
    _, delta = ops.feature_forward(z, C, LO, HI, G, "identity", 1.0, delta_f32=True, **kw)
    for rows in (slice(0, 8), slice(N - 8, N)):
        _, ref = util.oc.feature_forward(util.f32(z[rows]), util.f32(C), LO, HI, G, "identity", 1.0, spline_order=order)
        util.assert_parity("delta", delta[rows], ref, torch.float32, rel_gate=5e-6)
    _, dC, _ = ops.feature_backward(z, C, g, LO, HI, G, "identity", 1.0, need_dz=False, cast_dC=False, **kw)
    for keys in (slice(0, 4), slice(h - 4, h)):
        util.assert_parity("dC", dC[keys], _dC_of(z, C, g, G, order, keys), torch.float32, bias=True, rel_gate=5e-6)
    ops.check_status(z.device)


# one CTA per slab or more slabs than SMs, so that a run has all the tiles: on both sides of 16 and 32 tiles of 64 tokens
@pytest.mark.parametrize("N", [1023, 1024, 1025, 2048, 2049, 2113])
def test_dC_at_the_ends_of_its_segments(N):
    h, r, G = 12008, 16, 20
    z, g = _normal(N, h, seed=4), _normal(N, r, seed=5)
    C = torch.zeros(h, G + 1, r, dtype=torch.bfloat16, device="cuda")
    _, dC, dC_cast = ops.feature_backward(z, C, g, LO, HI, G, "identity", 1.0, with_base=False, need_dz=False, impl="tcgen05",
                                          spline_order=1)
    for keys in (slice(0, 4), slice(6000, 6004), slice(h - 4, h)):
        util.assert_parity("dC", dC[keys], _dC_of(z, C, g, G, 1, keys), torch.float32, bias=True, rel_gate=5e-6)
    assert torch.equal(dC_cast, dC.bfloat16())
    ops.check_status(z.device)


# a tile of 384 tokens for each of 148 SMs, so that one split has all the keys: on both sides of 8, 16 and 24 chunks of 8
@pytest.mark.parametrize("h", [57, 64, 65, 72, 128, 129, 192, 193])
def test_forward_at_the_ends_of_its_chains(h):
    N, r, G = 148 * 384 - 3, 20, 12
    z = _normal(N, h, seed=6)
    C = _normal(h, G + 2, r, seed=7) * 0.02
    a, delta = ops.feature_forward(z, C, LO, HI, G, "identity", 1.0, delta_f32=True, impl="tcgen05")
    assert torch.equal(a, z)
    for rows in (slice(0, 64), slice(N // 2, N // 2 + 64), slice(N - 64, N)):
        _, ref = util.oc.feature_forward(util.f32(z[rows]), util.f32(C), LO, HI, G, "identity", 1.0)
        util.assert_parity("delta", delta[rows], ref, torch.float32, rel_gate=5e-6)
    ops.check_status(z.device)
