"""Residual blocks of the UNet and the autoencoder with their biases folded into the ops around the convolutions: the same
values and gradients as the plain sequence, and every hook or replaced module is still called."""
import pytest
import torch
import torch.nn as nn

from eridiffusion_b200.models.sdxl_unet import ResBlock, SDXLConfig
from eridiffusion_b200.models.vae import _Res
from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu
KW = dict(device="cuda", dtype=torch.bfloat16)


def randomised(m, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(torch.randn(p.shape, device="cuda", generator=g) * (0.5 if p.dim() == 1 else (2 / p[0].numel()) ** 0.5))
    return m


def nhwc(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)


class Doubled(nn.Linear):
    def forward(self, x):
        return 2 * super().forward(x)


@pytest.mark.parametrize("what", ["temb hook", "temb pre-hook", "temb replaced", "temb backward hook", "temb forward"])
def test_time_embedding_module_is_called(what):
    torch.manual_seed(0)
    blk = randomised(ResBlock(64, 64, 128, SDXLConfig(), torch.bfloat16, "cuda"))
    x, emb = nhwc(2, 64, 8, 8).requires_grad_(), torch.randn(2, 128, **KW)
    plain = blk(x, emb)
    seen = []
    if what == "temb hook":
        blk.temb.register_forward_hook(lambda m, a, y: seen.append(y) or 2 * y)
    elif what == "temb pre-hook":
        blk.temb.register_forward_pre_hook(lambda m, a: seen.append(a) or (a[0] * 0,))
    elif what == "temb backward hook":
        blk.temb.register_full_backward_hook(lambda m, gi, go: seen.append(go))
    elif what == "temb forward":
        fwd = blk.temb.forward
        blk.temb.forward = lambda t: seen.append(t) or 2 * fwd(t)
    else:
        old, blk.temb = blk.temb, Doubled(128, 64, **KW)
        blk.temb.load_state_dict(old.state_dict())
    y = blk(x, emb)
    y.sum().backward()
    assert seen or what == "temb replaced"
    # (a listener that changes nothing: one bf16 rounding of the embedding may fall the other way)
    near = (y - plain).abs().max() <= 2.0 ** -5 * plain.abs().max()
    assert near if what == "temb backward hook" else not near


@pytest.mark.parametrize("name", ["conv1", "conv2", "skip", "norm2"])
@pytest.mark.parametrize("kind", ["forward", "pre", "backward", "backward pre"])
def test_hooks_of_a_unet_block_fire(name, kind):
    blk = randomised(ResBlock(64, 128, 128, SDXLConfig(), torch.bfloat16, "cuda"))
    seen, m = [], getattr(blk, name)
    reg = {"forward": m.register_forward_hook, "pre": m.register_forward_pre_hook, "backward": m.register_full_backward_hook,
           "backward pre": m.register_full_backward_pre_hook}[kind]
    reg(lambda m, *a: seen.append(a) and None)
    blk(nhwc(2, 64, 8, 8).requires_grad_(), torch.randn(2, 128, **KW)).sum().backward()
    assert len(seen) == 1
    if kind == "pre":
        assert len(seen[0][0]) == 1         # the module's own call, without addends


@pytest.mark.parametrize("name", ["c1", "c2", "n1", "n2"])
def test_hooks_of_an_autoencoder_block_fire(name):
    blk, seen = randomised(_Res(64, 64, 32, KW)), []
    getattr(blk, name).register_full_backward_hook(lambda *a: seen.append(a) and None)
    blk(nhwc(2, 64, 8, 8).requires_grad_()).sum().backward()
    assert len(seen) == 1
