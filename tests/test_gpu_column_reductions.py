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


@pytest.mark.parametrize("Nn,H,W,C", [(1, 2, 2, 32), (2, 7, 9, 320), (1, 65, 64, 128), (3, 8, 8, 1280)])
def test_conv_companions(Nn, H, W, C):
    """The bias of a convolution and a per-sample embedding added inside the norm, the residual sum with two biases,
    and upsampling, forward and backward, on channels-last activations."""
    def nhwc(seed):
        return rnd(Nn, H, W, C, seed=seed).permute(0, 3, 1, 2)
    x = nhwc(1).detach().requires_grad_()
    w, b = (rnd(C, seed=2, scale=0.3) + 1).requires_grad_(), rnd(C, seed=3).requires_grad_()
    pc, pn = rnd(C, seed=4).requires_grad_(), rnd(Nn, C, seed=5).requires_grad_()
    pc.grad = torch.ones_like(pc)                    # added into an existing gradient
    dy = nhwc(6)
    y = F.group_norm_silu(x, w, b, 32, 1e-5, True, pc, pn)
    y.backward(dy)
    ref = [t.detach().float().requires_grad_() for t in (x, w, b, pc, pn)]
    xr, wr, br, pcr, pnr = ref
    z = torch.nn.functional.group_norm(xr + pcr[:, None, None] + pnr[:, :, None, None], 32, wr, br, 1e-5)
    yr = torch.nn.functional.silu(z)
    yr.backward(dy.float())
    assert y.is_contiguous(memory_format=torch.channels_last)
    # dx sums to nearly zero over a group, so the gradients of the addends are compared against the size of dx's sums
    scale = xr.grad.abs().sum((2, 3)).max().item()
    for got, want, tol in ((y, yr, yr.abs().max().item()), (x.grad, xr.grad, xr.grad.abs().max().item()),
                           (w.grad, wr.grad, wr.grad.abs().max().item()), (b.grad, br.grad, br.grad.abs().max().item()),
                           (pn.grad, pnr.grad, scale), (pc.grad, pcr.grad + 1, Nn * scale + 1)):
        assert (got.float() - want).abs().max().item() <= 1e-2 * tol
    a, c = nhwc(7).detach().requires_grad_(), nhwc(8).detach().requires_grad_()
    b1, b2 = rnd(C, seed=9).requires_grad_(), rnd(C, seed=10).requires_grad_()
    out = F.add_bias(a, c, b1, b2)
    out.backward(dy)
    want = a.float() + c.float() + b1.float()[:, None, None] + b2.float()[:, None, None]
    assert (out.float() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item()
    assert torch.equal(a.grad, dy) and torch.equal(b1.grad, b2.grad)
    close_sum(b1.grad, dy.double().sum((0, 2, 3)), Nn * H * W)
    u = nhwc(11).detach().requires_grad_()
    up = F.upsample2x(u)
    assert torch.equal(up, torch.nn.functional.interpolate(u, scale_factor=2.0, mode="nearest"))
    du = rnd(Nn, 2 * H, 2 * W, C, seed=12).permute(0, 3, 1, 2)
    up.backward(du)
    want = du.float().view(Nn, C, H, 2, W, 2).sum((3, 5))
    assert (u.grad.float() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item()


@pytest.mark.parametrize("B,L,Lk,H,D", [(1, 16, 16, 2, 64), (2, 130, 77, 3, 64), (1, 257, 300, 2, 128), (2, 128, 1, 1, 128)])
def test_packed_attention(B, L, Lk, H, D):
    """q, k and v read inside the projections' outputs, gradients written as packed tensors."""
    qkv = rnd(B, L, 3 * H * D, seed=1).requires_grad_()
    o = F.attention_qkv(qkv, H)
    q, k, v = (t.contiguous() for t in qkv.detach().view(B, L, 3, H, D).unbind(2))
    ref = [t.requires_grad_() for t in (q, k, v)]
    orf = F.attention(*ref).reshape(B, L, H * D)
    do = rnd(B, L, H * D, seed=2)
    o.backward(do)
    orf.backward(do)
    assert torch.equal(o, orf)                       # the same kernels on the same values
    assert torch.equal(qkv.grad.view(B, L, 3, H, D), torch.stack([t.grad for t in ref], 2))
    qq, kv = rnd(B, L, H * D, seed=3).requires_grad_(), rnd(B, Lk, 2 * H * D, seed=4).requires_grad_()
    o = F.attention_kv(qq, kv, H)
    k, v = (t.contiguous() for t in kv.detach().view(B, Lk, 2, H, D).unbind(2))
    ref = [t.requires_grad_() for t in (qq.detach().view(B, L, H, D), k, v)]
    orf = F.attention(*ref).reshape(B, L, H * D)
    o.backward(do)
    orf.backward(do)
    assert torch.equal(o, orf) and torch.equal(qq.grad.view(B, L, H, D), ref[0].grad)
    assert torch.equal(kv.grad.view(B, Lk, 2, H, D), torch.stack([ref[1].grad, ref[2].grad], 2))


@pytest.mark.parametrize("n", [1, 7, 8, 1023, 2048, 4099])
@pytest.mark.parametrize("off", [0, 1])
def test_weight_average_sizes(n, off):
    p = rnd(n + off, seed=1)[off:]
    s0 = torch.randn(n + off, device="cuda")[off:]
    s = s0.clone() if off == 0 else torch.empty(n + 1, device="cuda")[1:].copy_(s0)
    N.check(N.require().eri_ema_update(s.data_ptr(), p.data_ptr(), n, 0.9, N.stream_ptr()), "ema")
    want = 0.9 * s0.double() + (1 - 0.9) * p.double()
    assert (s.double() - want).abs().max().item() <= 1e-6 * want.abs().max().item() + 1e-6
