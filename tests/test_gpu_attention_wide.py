"""Attention at head size 512 (image autoencoders) against fp64: token counts around the 128-row tiles of queries and keys,
column blocks of a packed projection, several heads and batches."""
import pytest
import torch

from eridiffusion_b200.ops import flash_attn as FA
from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _ref(q, k, v, scale):
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    return (torch.softmax(q @ k.transpose(-1, -2) * scale, -1) @ v).transpose(1, 2)


@pytest.mark.parametrize("B,Lq,Lk,H,packed,spread", [(1, 128, 128, 1, True, 1.0), (1, 129, 129, 1, True, 1.0), (2, 200, 200, 2, True, 3.0),
                                                     (1, 255, 385, 1, False, 1.0), (1, 640, 640, 1, True, 8.0), (1, 1000, 130, 3, False, 8.0)])
def test_wide_attention(B, Lq, Lk, H, packed, spread):
    g = torch.Generator(device="cuda").manual_seed(Lq + Lk)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    if packed:
        q, k, v = mk(B, Lq, 3, H, 512).unbind(2)
    else:
        q, k, v = mk(B, Lq, H, 512), mk(B, Lk, H, 512), mk(B, Lk, H, 512)
    scale = spread / 512 ** 0.5            # wide spreads move the running maximum: the rescaling path
    calls = F.ATTENTION_CALLS["native"]
    o = F.attention(q, k, v, scale)
    assert F.ATTENTION_CALLS["native"] == calls + 1 and FA.check_error() == 0
    r = _ref(q, k, v, scale)
    # probabilities and results rounded to bf16 once each (2^-9 relative)
    assert ((o.double() - r).norm() / r.norm()).item() < 2 ** -7
    assert ((o.double() - r).abs().max() / r.abs().max()).item() < 2 ** -6


@pytest.mark.parametrize("L,grad", [(127, False), (256, True)])
def test_calls_beyond_the_kernel_keep_their_answer(L, grad):
    q, k, v = (torch.randn(1, L, 1, 512, device="cuda", dtype=torch.bfloat16, requires_grad=grad) for _ in range(3))
    o = F.attention(q, k, v)
    r = _ref(q.detach(), k.detach(), v.detach(), 512 ** -0.5)
    assert ((o.double() - r).norm() / r.norm()).item() < 2 ** -6
    if grad:
        o.float().sum().backward()
        assert torch.isfinite(q.grad).all() and v.grad.abs().sum() > 0
