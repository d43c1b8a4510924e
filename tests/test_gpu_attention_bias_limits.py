"""Attention with a mask per query and key at the limits of the mask's type, against fp64: the lowest finite value hides a key
only next to a visible one, -inf and False always do."""
import pytest
import torch

from eridiffusion_b200.ops import flash_attn as FA
from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu
LOW = torch.finfo(torch.bfloat16).min


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Lk", [64, 131, 300])          # vector and scalar mask rows, one to three key tiles
@pytest.mark.parametrize("kind", ["rows", "first tile", "causal", "nearly lowest", "inf rows", "inf and lowest", "bool rows"])
def test_mask_limits(kind, Lk, D):
    B, Lq, H = 1, 140, 2
    g = torch.Generator(device="cuda").manual_seed(Lk + D)
    q, k, v = (torch.randn(B, n, H, D, device="cuda", generator=g).to(torch.bfloat16) for n in (Lq, Lk, Lk))
    m = torch.zeros(1, 1, Lq, Lk, device="cuda", dtype=torch.bfloat16)
    if kind == "rows":
        m[..., ::3, :] = LOW
    elif kind == "first tile":
        m[..., :128] = LOW
    elif kind == "causal":
        m = torch.full_like(m, LOW).triu(1)
    elif kind == "nearly lowest":           # the one key that is less hidden than the others takes everything
        m[:] = LOW
        m[..., Lk - 2] = -3.0e38
    elif kind == "inf rows":
        m[..., ::3, :] = float("-inf")
    elif kind == "inf and lowest":
        m[:] = float("-inf")
        m[..., 5:9] = LOW
    else:
        m = torch.ones_like(m, dtype=torch.bool)
        m[..., ::3, :] = False
    s = q.double().transpose(1, 2) @ k.double().transpose(1, 2).transpose(-1, -2) * D ** -0.5
    s = s.masked_fill(~m, float("-inf")) if m.dtype == torch.bool else s + m.double()
    r = (torch.softmax(s, -1).nan_to_num(0.0) @ v.double().transpose(1, 2)).transpose(1, 2)
    o = F.attention(q, k, v, mask=m)
    assert FA.check_error() == 0 and torch.isfinite(o).all()
    # fp32 inside, one rounding of the result to bf16 (2^-9 of each value)
    assert ((o.double() - r).abs() <= 2.0 ** -8 * r.abs() + 2.0 ** -14).all()
