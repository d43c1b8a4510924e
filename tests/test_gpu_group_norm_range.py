"""GroupNorm at the ends of its range: channel counts around the 640- and 1024-thread kernels, many groups, many chunks."""
import pytest
import torch

from eridiffusion_b200.ops import _native as N
from eridiffusion_b200.ops import functional as F
from eridiffusion_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def rnd(*s, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*s, device="cuda", generator=g) * scale).bfloat16()


@pytest.mark.parametrize("Nn,HW,C,G", [(1, 30, 5120, 32), (2, 30, 5128, 8), (1, 700, 6144, 32), (1, 9, 8192, 512), (1, 40, 8192, 4096),
                                       (1, 4099, 1024, 1024), (2, 77, 2048, 1024)])
@pytest.mark.parametrize("pre", [False, True])
def test_wide_and_many_groups(Nn, HW, C, G, pre):
    x, w, b = rnd(Nn, HW, C, seed=1).requires_grad_(), (rnd(C, seed=2, scale=0.3) + 1).requires_grad_(), rnd(C, seed=3).requires_grad_()
    dy = rnd(Nn, HW, C, seed=4)
    pc, pn = (rnd(C, seed=5).requires_grad_(), rnd(Nn, C, seed=6).requires_grad_()) if pre else (None, None)
    n0 = N.launch_count()
    y = F.group_norm_silu(x, w, b, G, 1e-5, True, pc, pn)
    assert N.launch_count() > n0                     # on the kernels
    y.backward(dy)
    leaves = [t.detach().float().requires_grad_() for t in (x, w, b) + ((pc, pn) if pre else ())]
    z = leaves[0] + leaves[3] + leaves[4][:, None] if pre else leaves[0]
    yr = R.group_norm_silu(z, leaves[1], leaves[2], G, 1e-5, True)
    yr.backward(dy.float())
    for got, ref in ((y, yr), (x.grad, leaves[0].grad), (w.grad, leaves[1].grad), (b.grad, leaves[2].grad)):
        assert (got.float() - ref.detach()).abs().max().item() <= 1e-2 * ref.abs().max().item()
    if pre:             # sums of dx that nearly cancel: against the size of their terms
        scale = leaves[0].grad.abs().sum(1).max().item()
        assert (pn.grad.float() - leaves[4].grad).abs().max().item() <= 1e-2 * scale
        assert (pc.grad.float() - leaves[3].grad).abs().max().item() <= 1e-2 * Nn * scale


@pytest.mark.parametrize("value", [1e20, -3e30, float("inf"), float("nan")])
def test_overflowing_groups_are_not_finite_garbage(value):
    """Squares beyond fp32's range cannot be normalised: NaN, never a finite value; the other groups are untouched."""
    x = rnd(1, 64, 256, seed=1)
    w, b = torch.ones(256, device="cuda").bfloat16(), torch.zeros(256, device="cuda").bfloat16()
    clean = F.group_norm_silu(x, w, b, 32, silu=False)
    x[..., :8] = value
    y = F.group_norm_silu(x, w, b, 32, silu=False)
    assert y[..., :8].isnan().all() and torch.equal(y[..., 8:], clean[..., 8:])
