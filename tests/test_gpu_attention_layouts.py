"""Attention operands in every layout that callers hand over give what contiguous copies give, bit for bit, on the kernels."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def mk(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


def same_as_contiguous(q, k, v, **kw):
    def run(ts):
        ts = [t.detach().requires_grad_() for t in ts]
        n = F.ATTENTION_CALLS["native"]
        o = F.attention(*ts, **kw)
        assert F.ATTENTION_CALLS["native"] == n + 1
        o.backward(do)
        return o, [t.grad for t in ts]
    do = mk(*q.shape)
    o, g = run((q, k, v))
    oc, gc = run([torch.empty(t.shape, device="cuda", dtype=t.dtype).copy_(t) for t in (q, k, v)])
    assert torch.equal(o, oc) and all(torch.equal(a, b) for a, b in zip(g, gc))
    with torch.no_grad():
        assert torch.equal(F.attention(q, k, v, **kw), oc)


@pytest.mark.parametrize("D", [64, 128])
def test_dimensions_of_size_one(D):
    one_head = [mk(2, 1, 256, D).transpose(1, 2) for _ in range(3)]
    assert one_head[0].is_contiguous() and one_head[0].stride(2) != D
    same_as_contiguous(*one_head)
    same_as_contiguous(mk(2, 32, 4, D), *(mk(2, 4, 1, D).transpose(1, 2) for _ in "kv"))       # one key
    same_as_contiguous(*(mk(256, 1, 4, D).transpose(0, 1) for _ in "qkv"))                      # one sample
    same_as_contiguous(mk(1, 32, 1, D), *(mk(1, 1, 1, D).expand(1, 1, 1, D) for _ in "kv"))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H", [1, 3])
@pytest.mark.parametrize("masked", [False, True])
def test_column_blocks_and_transposed_views(D, H, masked):
    kw = dict(mask=torch.rand(2, 1, 1, 140, device="cuda") > 0.3) if masked else {}
    same_as_contiguous(*mk(2, 140, 3, H, D).unbind(2), **kw)                                # a packed projection
    same_as_contiguous(*(mk(2, H, 140, D).transpose(1, 2) for _ in "qkv"), **kw)            # head-major tensors
    same_as_contiguous(*(mk(2, 140, H, D + 1)[..., 1:] for _ in "qkv"), **kw)               # rows that are not aligned
    wide = mk(2, 140, H, 2 * D)
    same_as_contiguous(wide[..., :D], mk(2, 140, H, D), wide[..., D:], **kw)


def test_autoencoder_and_encoder_attention_stay_on_the_kernels():
    """Callers hand over views of the packed projection: head size 64 without a mask, and with a key mask."""
    from eridiffusion_b200.models.vae import _Attn
    n = dict(F.ATTENTION_CALLS)
    _Attn(64, 32, dict(device="cuda", dtype=torch.bfloat16))(mk(1, 64, 16, 16).contiguous(memory_format=torch.channels_last))
    assert F.ATTENTION_CALLS["native"] == n["native"] + 1 and F.ATTENTION_CALLS["library"] == n["library"]


@pytest.mark.parametrize("scale", [-2.0, -0.1, 0.0, 2.0])
def test_head_512_with_any_scale(scale):
    q, k, v = mk(1, 160, 1, 512), mk(1, 192, 1, 512), mk(1, 192, 1, 512)
    o = F.attention(q, k, v, scale=scale)
    r = F.R.attention_fp32(q.double(), k.double(), v.double(), scale)
    # bf16 probabilities and one rounding of the result: 2^-8 of values of order one to four
    assert torch.isfinite(o).all() and (o.float() - r).abs().max().item() < 2.0 ** -5
