"""Column reductions (bias, norm-parameter, modulation and gate gradients) and the two-pass GroupNorm at the edges of
their tiles: row counts below one lane group, column counts that leave a partial 64-column CTA, chunk counts on both
sides of the fold."""
import pytest
import torch

from eridiffusion_b200.ops import _native as N
from eridiffusion_b200.ops import functional as F
from eridiffusion_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def rnd(*s, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*s, device="cuda", generator=g) * scale).bfloat16()


def close_sum(got, ref, terms):
    # fp32 sums of `terms` products, then one rounding to bf16 (2^-9 relative)
    tol = 2.0 ** -8 * ref.abs().max().item() + terms * 2.0 ** -23 * ref.abs().max().item()
    assert (got.float() - ref).abs().max().item() <= tol


@pytest.mark.parametrize("B,L,D", [(1, 1, 8), (1, 77, 72), (2, 257, 320), (3, 1000, 264), (1, 4096, 3072)])
def test_column_reductions(B, L, D):
    x, dy = rnd(B, L, D, seed=1), rnd(B, L, D, seed=2)
    bias = rnd(D, seed=3).requires_grad_()
    xd, dd = x.double(), dy.double()
    # sum: through a linear's bias, returned and accumulated
    w = rnd(D, 64, seed=4, scale=0.1)
    xin = rnd(1, B * L, 64, seed=5)
    for acc in (False, True):
        bias.grad = torch.ones_like(bias) if acc else None
        F.linear(xin, w, bias).backward(dy.view(1, B * L, D))
        close_sum(bias.grad, dd.sum((0, 1)) + (1.0 if acc else 0.0), B * L)
    # norm: affine over all rows, modulation per batch element
    if D >= 256:
        wt, bs = rnd(D, seed=6).requires_grad_(), rnd(D, seed=7).requires_grad_()
        F.norm_modulate(x, weight=wt, bias=bs, eps=1e-5).backward(dy)
        xh = (xd - xd.mean(-1, keepdim=True)) / (xd.var(-1, unbiased=False, keepdim=True) + 1e-5).sqrt()
        close_sum(bs.grad, dd.sum((0, 1)), B * L)
        assert (wt.grad.double() - (dd * xh).sum((0, 1))).abs().max() <= 1e-2 * (dd * xh).sum((0, 1)).abs().max()
        sc, sh = rnd(B, D, seed=8, scale=0.3).requires_grad_(), rnd(B, D, seed=9).requires_grad_()
        F.norm_modulate(x, sc, sh, eps=1e-5).backward(dy)
        close_sum(sh.grad, dd.sum(1), L)
        assert (sc.grad.double() - (dd * xh).sum(1)).abs().max() <= 1e-2 * (dd * xh).sum(1).abs().max()
    # dot: the gate's gradient
    gate = rnd(B, D, seed=10).requires_grad_()
    F.gate_residual(None, x, gate).backward(dy)
    close_sum(gate.grad, (dd * xd).sum(1), L)


@pytest.mark.parametrize("Nn,HW,C,G", [(1, 2, 32, 32), (2, 63, 320, 32), (1, 64 * 64 + 3, 128, 32), (3, 1024, 1280, 32),
                                       (1, 40, 5120, 32), (2, 100, 2560, 16)])
@pytest.mark.parametrize("silu", [False, True])
def test_group_norm_passes(Nn, HW, C, G, silu):
    x = rnd(Nn, HW, C, seed=1).requires_grad_()
    w, b = (rnd(C, seed=2, scale=0.3) + 1).requires_grad_(), rnd(C, seed=3).requires_grad_()
    dy = rnd(Nn, HW, C, seed=4)
    w.grad = torch.ones_like(w)                      # added into an existing gradient; b gets a new one
    y = F.group_norm_silu(x, w, b, G, 1e-5, silu)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = R.group_norm_silu(xr, wr, br, G, 1e-5, silu)
    yr.backward(dy.float())
    for got, ref in ((y, yr), (x.grad, xr.grad), (w.grad, wr.grad + 1), (b.grad, br.grad)):
        assert (got.float() - ref.detach()).abs().max().item() <= 1e-2 * ref.abs().max().item()
    y2 = F.group_norm_silu(x, w, b, G, 1e-5, silu)
    assert torch.equal(y, y2)                        # the sums do not depend on timing
    assert N.launch_count() > 0
