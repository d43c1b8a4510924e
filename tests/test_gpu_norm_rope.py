"""Self-attention on a packed projection with a full-width QK-norm and rotary embedding: the fused kernels against the
fp64 composition of the same definition."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _reference(qkv, wq, wk, cos, sin, H, eps):
    B, L, W = qkv.shape
    D = W // 3
    q, k, v = qkv.split(D, dim=-1)

    def nr(t, w):
        t = t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + eps) * w
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack((cos * a - sin * b, sin * a + cos * b), -1).flatten(-2).view(B, L, H, D // H)
    q, k, v = nr(q, wq), nr(k, wk), v.reshape(B, L, H, D // H)
    p = torch.softmax(torch.einsum("blhd,bmhd->bhlm", q, k) * (D // H) ** -0.5, -1)
    return torch.einsum("bhlm,bmhd->blhd", p, v).reshape(B, L, D)


# widths on both sides of each vectors-per-thread step (2048, 4096, 8192), token counts around one attention tile
@pytest.mark.parametrize("B,L,H,Dh,shift", [(1, 16, 2, 64, 0), (2, 77, 16, 128, 0), (1, 129, 33, 64, 0), (1, 200, 32, 128, 0),
                                            (1, 40, 33, 128, 0), (1, 130, 64, 128, 0), (2, 33, 4, 64, 4)])
def test_norm_rope_attention(B, L, H, Dh, shift):
    D = H * Dh
    g = torch.Generator(device="cuda").manual_seed(B * L + D)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    base = torch.empty(B * L * 3 * D + shift, device="cuda", dtype=torch.bfloat16)
    base.copy_(mk(base.numel()))
    qkv = base[shift:].view(B, L, 3 * D).requires_grad_()          # shift: not on a 16-byte boundary
    wq, wk = (1 + 0.1 * mk(2, D)).to(torch.bfloat16)
    ang = mk(L, D // 2 + 4)                                        # tables with a row stride of their own
    cos, sin = torch.cos(ang)[:, :D // 2], torch.sin(ang)[:, :D // 2]
    dy = mk(B, L, D).to(torch.bfloat16)
    calls = F.ATTENTION_CALLS["native"]
    y = F.attention_qkv_rope(qkv, wq, wk, cos, sin, H)
    assert F.ATTENTION_CALLS["native"] == calls + 1
    (d,) = torch.autograd.grad(y, qkv, dy)
    with torch.no_grad():
        assert torch.equal(F.attention_qkv_rope(qkv, wq, wk, cos, sin, H), y)
    x64 = qkv.detach().double().requires_grad_()
    y64 = _reference(x64, wq.double(), wk.double(), cos.double(), sin.double(), H, 1e-6)
    (d64,) = torch.autograd.grad(y64, x64, dy.double())
    # bf16 operands, probabilities and results, each rounded once (2^-9 relative, random signs): under 2^-7 together
    for a, b in ((y, y64), (d[..., 2 * D:], d64[..., 2 * D:]), (d[..., :D], d64[..., :D]), (d[..., D:2 * D], d64[..., D:2 * D])):
        assert ((a.double() - b).norm() / b.norm()).item() < 2 ** -6


def test_trainable_norm_weights_keep_their_gradient():
    D, H = 128, 2
    w = [torch.ones(D, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2)]
    qkv = torch.randn(1, 32, 3 * D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    t = torch.rand(32, D // 2, device="cuda")
    F.attention_qkv_rope(qkv, *w, torch.cos(t), torch.sin(t), H).float().square().sum().backward()
    assert all(x.grad is not None and x.grad.abs().sum() > 0 for x in (*w, qkv))
