"""Calls of the CUDA-core kernels behind one another on a stream, each reading what the one before it writes (their first kernel is
chained to that call's last and starts early): bit for bit what the same calls give with the GPU waited for in between."""
import pytest
import torch

from tests import util

pytestmark = pytest.mark.gpu

ops = pytest.importorskip("sparsespline_ffn_b200.ops")

F32, BF16 = torch.float32, torch.bfloat16
STEPS, REPEATS = 8, 10


def _forwards(z, C, outs, impl, wait):
    r = C.shape[2]
    for f in outs:
        ops.feature_forward(z, C, -3.0, 3.0, C.shape[1] - 2, "identity", 0.75, impl=impl, out=f)
        z = f[:, r:]                                  # columns of phi(z) and of delta, read in place
        if wait:
            torch.cuda.synchronize()


@pytest.mark.parametrize("N,h,r,dtype,impl", [
    (1, 5120, 32, BF16, "auto"),       # a cluster of CTAs per token
    (64, 512, 64, F32, "auto"),
    (40, 96, 20, F32, "auto"),         # rows that are read element by element
    (700, 512, 32, F32, "auto"),       # key splits, added by a kernel of their own
    (20000, 64, 32, F32, "auto"),      # one split
    (3000, 256, 32, BF16, "simt"),
])
def test_forwards_behind_one_another(N, h, r, dtype, impl):
    C = (torch.randn(h, 22, r, generator=torch.Generator().manual_seed(3)) * 0.1).to(dtype).cuda()
    outs, refs = ([torch.empty(N, h + r, dtype=dtype, device="cuda") for _ in range(STEPS)] for _ in range(2))
    for seed in range(REPEATS):
        z = util.make_inputs(N, h, r, 20, dtype, seed=seed)[0]
        _forwards(z, C, refs, impl, True)
        for f in outs:
            f.fill_(1e3)
        _forwards(z, C, outs, impl, False)
        for f, ref in zip(outs, refs):
            assert torch.equal(f, ref)


def _backwards(zs, Cs, go, wait):
    got = []
    for z, C in zip(zs, Cs):
        dz, dC, _ = ops.feature_backward(z, C, go, -3.0, 3.0, C.shape[1] - 2, "gelu", 0.75, impl="simt")
        got += [dz, dC]
        go = dz                                       # [N, h] of this layer is [N, h + r] of the next
        if wait:
            torch.cuda.synchronize()
    return got


@pytest.mark.parametrize("N,h,r,dtype", [(513, 288, 32, F32), (4096, 288, 32, F32), (300, 180, 20, F32), (1000, 288, 32, BF16)])
def test_backwards_behind_one_another(N, h, r, dtype):
    widths = [h - r * k for k in range(6)]
    gen = torch.Generator().manual_seed(5)
    zs = [torch.randn(N, w, generator=gen).to(dtype).cuda() for w in widths]
    Cs = [(torch.randn(w, 22, r, generator=gen) * 0.1).to(dtype).cuda() for w in widths]
    for _ in range(REPEATS):
        go = torch.randn(N, h + r, generator=gen).to(dtype).cuda()
        refs = _backwards(zs, Cs, go, True)
        for got, ref in zip(_backwards(zs, Cs, go, False), refs):
            assert torch.equal(got, ref)


def test_captured_behind_a_copy_and_another_stream():
    """In a graph: the first call behind a copy, the second behind the first and behind work of a second stream."""
    N, h, r = 64, 512, 32
    C = (torch.randn(h, 22, r, generator=torch.Generator().manual_seed(3)) * 0.1).cuda()
    zin, z = (torch.zeros(N, h, device="cuda") for _ in range(2))
    f0, f1 = (torch.empty(N, h + r, device="cuda") for _ in range(2))
    go = torch.empty(N, h + r, device="cuda")
    side, joined = torch.cuda.Stream(), []

    def step():
        z.copy_(zin)
        _forwards(z, C, [f0], "auto", False)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.mul(z[:, :h], 2.0, out=go[:, :h])
            torch.mul(f0[:, h:], 3.0, out=go[:, h:])
        torch.cuda.current_stream().wait_stream(side)
        joined[:] = ops.feature_backward(f0[:, r:], C, go, -3.0, 3.0, 20, "gelu", 0.75, impl="simt")[:2]
        _forwards(f0[:, r:], C, [f1], "auto", False)

    step()                                            # before the capture: kernels loaded, scratch in the pool
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    held = list(joined)
    for seed in range(REPEATS):
        zin.copy_(util.make_inputs(N, h, r, 20, F32, seed=seed)[0])
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (f0, f1, *held)]
        step()
        torch.cuda.synchronize()
        for a, b in zip(got, (f0, f1, *joined)):
            assert torch.equal(a, b)
