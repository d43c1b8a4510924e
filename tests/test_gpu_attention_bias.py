"""Attention with a mask per query and key against fp64: broadcasts, boolean and additive masks, rows without a visible key,
token counts around the 128-row tiles, unaligned mask rows."""
import pytest
import torch

from eridiffusion_b200.ops import flash_attn as FA
from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _ref(q, k, v, mask, scale):
    s = q.double().transpose(1, 2) @ k.double().transpose(1, 2).transpose(-1, -2) * scale
    s = s.masked_fill(~mask, float("-inf")) if mask.dtype == torch.bool else s + mask.double()
    p = torch.softmax(s, -1).nan_to_num(0.0)
    return (p @ v.double().transpose(1, 2)).transpose(1, 2)


@pytest.mark.parametrize("B,Lq,Lk,H,D,shape", [(2, 77, 77, 12, 64, "causal"), (1, 256, 256, 4, 64, "hqk"), (3, 130, 130, 2, 64, "bhqk"),
                                               (2, 64, 300, 3, 128, "bqk"), (1, 1, 5, 1, 128, "hqk"), (2, 257, 129, 2, 64, "blind"),
                                               (1, 384, 384, 2, 64, "spread"), (2, 200, 136, 2, 128, "sliced")])
def test_bias_attention(B, Lq, Lk, H, D, shape):
    g = torch.Generator(device="cuda").manual_seed(Lq + Lk)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    if Lq == Lk:
        q, k, v = mk(B, Lq, 3, H, D).unbind(2)
    else:
        q, k, v = mk(B, Lq, H, D), mk(B, Lk, H, D), mk(B, Lk, H, D)
    scale = D ** -0.5
    if shape == "causal":
        mask = torch.ones(Lq, Lk, dtype=torch.bool, device="cuda").tril()[None, None]
    elif shape == "blind":               # the first keys, and for some queries all keys, are hidden
        mask = torch.rand(B, 1, Lq, Lk, device="cuda", generator=g) > 0.5
        mask[..., :100] = False
        mask[:, :, ::3] = False
    elif shape == "sliced":
        mask = mk(B, H, Lq, Lk + 3)[..., 1:Lk + 1]
    else:
        mask = mk(B if "b" in shape else 1, H if "h" in shape else 1, Lq, Lk)
        if shape == "spread":            # the running maximum moves: the rescaling path
            mask = mask * 20
        if "b" in shape:
            mask[:, :, :, -4:] = -1e4
    with torch.no_grad():
        lib = F.R.attention(q, k, v, scale, mask)
    r = _ref(q, k, v, mask, scale)
    key_only = mask.shape[1] == mask.shape[2] == 1
    calls = F.ATTENTION_CALLS["native"]
    o = F.attention(q, k, v, scale, mask)
    assert F.ATTENTION_CALLS["native"] == calls + 1 and FA.check_error() == 0
    if key_only:                         # a mask of keys alone keeps its own kernel (bf16 probabilities)
        return
    # fp32 throughout (probabilities as three bf16 terms): what is left is one rounding of the result to bf16, 2^-9
    assert ((o.double() - r).norm() / r.norm()).item() < 2 ** -8.5
    e0, e1 = ((t.double() - r).norm().item() for t in (lib, o))
    assert e1 <= e0 * 1.02
    if shape == "blind":
        assert (o[:, ::3] == 0).all()
