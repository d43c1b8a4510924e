"""Gradients that the kernels add straight into existing buffers: only in a plain backward pass, never where the caller asked
for the gradient itself or listens to the parameter."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _case(kind):
    torch.manual_seed(0)
    mk = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)  # noqa: E731
    if kind == "linear":
        ps = [mk(256, 128), mk(256)]
        x = mk(1, 300, 128).requires_grad_()
        return ps, lambda: F.linear(x, *ps).float().square().mean()
    if kind == "group_norm":
        ps = [mk(64), mk(64), mk(64)]
        x = mk(1, 200, 64).requires_grad_()
        return ps, lambda: F.group_norm_silu(x, ps[0], ps[1], 8, pre_c=ps[2]).float().square().mean()
    ps = [mk(256), mk(256)]
    x = mk(1, 300, 256).requires_grad_()
    return ps, lambda: F.norm_modulate(x, weight=ps[0], bias=ps[1]).float().square().mean()


@pytest.mark.parametrize("kind", ["linear", "group_norm", "norm"])
def test_asked_for_gradients_leave_the_buffers_alone(kind):
    ps, loss = _case(kind)
    for p in ps:
        p.requires_grad_()
        p.grad = torch.full_like(p, 3.0)
    want = torch.autograd.grad(loss(), ps)
    assert all((p.grad == 3).all() for p in ps) and all(w.abs().sum() > 0 for w in want)
    seen = []
    handles = [p.register_hook(lambda g: seen.append(g.clone())) for p in ps]
    loss().backward()
    assert len(seen) == len(ps)
    for h in handles:
        h.remove()
    hooked = [p.grad.clone() for p in ps]
    for p in ps:
        p.grad = torch.full_like(p, 3.0)
    loss().backward()
    for p, w, h in zip(ps, want, hooked):
        # one rounding of the sum to bf16 on either way, 2^-8 of the largest value
        tol = 2 ** -7 * (3 + w.abs().max().item())
        assert (p.grad - 3 - w).abs().max().item() <= tol and (h - 3 - w).abs().max().item() <= tol
