"""What autograd wraps around an operator: forward-mode tangents, tracing and saved-tensor hooks meet the native host path
as they met the Python autograd functions."""
import pytest
import torch


pytestmark = pytest.mark.gpu

fsf = pytest.importorskip("sparsespline_ffn_b200")

N, H, R, G = 200, 24, 16, 12


def _call(which, z, C):
    if which == "delta":
        return fsf.flash_spline_delta(z, C, -3.0, 3.0, G, 0.5)
    return fsf.flash_spline_feature(z, C, -3.0, 3.0, G, "relu_sq", 0.5, spline_order=1 if which == "linear" else 2)


def _inputs(which, dtype=torch.bfloat16):
    gen = torch.Generator().manual_seed(3)
    z = torch.randn(N, H, generator=gen).to(dtype).cuda()
    C = (torch.randn(H, G + (1 if which == "linear" else 2), R, generator=gen) * 0.1).to(dtype).cuda()
    go = torch.randn(N, R if which == "delta" else H + R, generator=gen).to(dtype).cuda()
    return z, C, go


@pytest.mark.parametrize("which", ["feature", "linear", "delta"])
def test_forward_mode_is_refused_and_not_dropped(which):
    # no jvp is defined: an error, never an output without its tangent
    z, C, _ = _inputs(which)
    with torch.autograd.forward_ad.dual_level():
        for a, b in ((torch.autograd.forward_ad.make_dual(z, torch.ones_like(z)), C),
                     (z, torch.autograd.forward_ad.make_dual(C, torch.ones_like(C)))):
            with pytest.raises(RuntimeError, match="jvp"):
                _call(which, a, b)


@pytest.mark.parametrize("which", ["feature", "linear", "delta"])
def test_a_traced_call_computes(which):
    z, C, _ = _inputs(which)
    traced = torch.jit.trace(lambda a, b: _call(which, a, b), (z, C), check_trace=False)
    z2, C2, _ = (t.flip(0).contiguous() for t in _inputs(which))
    assert torch.equal(traced(z2, C2), _call(which, z2, C2))


@pytest.mark.parametrize("change", ["same", "cpu", "columns first", "strided rows", "wider"])
@pytest.mark.parametrize("which", ["feature", "linear", "delta"])
def test_saved_tensors_come_back_in_another_form(which, change):
    def unpack(t):
        if change == "cpu":
            return t.cuda()
        if change == "columns first":
            return t.transpose(0, -1).contiguous().transpose(0, -1)
        if change == "strided rows":
            wide = torch.empty(*t.shape[:-1], t.shape[-1] + 8, dtype=t.dtype, device=t.device)
            wide[..., :t.shape[-1]] = t
            return wide[..., :t.shape[-1]]
        return t.float() if change == "wider" else t

    z, C, go = _inputs(which)
    want = []
    for hooked in (False, True):
        a, b = z.clone().requires_grad_(True), C.clone().requires_grad_(True)
        if hooked:
            with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu() if change == "cpu" else t, unpack):
                f = _call(which, a, b)
        else:
            f = _call(which, a, b)
        f.backward(go)
        want.append((f.detach(), a.grad, b.grad))
    for x, y in zip(*want):
        assert x.dtype == y.dtype and torch.equal(x, y)


def test_a_saved_tensor_of_another_shape_is_refused():
    z, C, go = _inputs("feature")
    a, b = z.clone().requires_grad_(True), C.clone().requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t[:-1] if t.dim() == 3 else t):
        f = fsf.flash_spline_feature(a, b, -3.0, 3.0, G, "relu_sq", 0.5)
    with pytest.raises((RuntimeError, ValueError)):
        f.backward(go)
