"""Residual blocks of the UNet and the autoencoder with their biases folded into the ops around the convolutions: the same
values and gradients as the plain sequence, and every hook or replaced module is still called."""
import copy

import pytest
import torch
import torch.nn as nn

from eridiffusion_b200.models.layers import channels_last_convs
from eridiffusion_b200.models.sdxl_unet import ResBlock, SDXLConfig
from eridiffusion_b200.models.vae import Encoder, VaeConfig, _Res, _run
from eridiffusion_b200.ops import functional as F
from eridiffusion_b200.optim import ParamArena

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


def gradients(m, call, dy):
    """Output, input gradients and every parameter's gradient of ``call(m)`` -> (output, inputs)."""
    for p in m.parameters():
        p.grad = None if p.grad is None else p.grad.zero_()
    y, ins = call(m)
    y.backward(dy.to(y.dtype))
    return {"out": y.detach(), **{f"in{i}": t.grad for i, t in enumerate(ins)}, **{n: p.grad for n, p in m.named_parameters()}}


def no_further_than_plain_bf16(m, call, arena):
    """The folded form, the plain bf16 sequence and fp32 on the same weights. Both bf16 forms round every activation and
    gradient (2^-9 each), in another order: their errors are two draws of the same size, of which one may be up to three
    times the other. A bias dropped, added twice or without its gradient is off by its own size, some hundred times that."""
    torch.manual_seed(0)
    ref, plain = copy.deepcopy(m).float(), copy.deepcopy(m)
    if arena == "arena":
        ParamArena(list(m.parameters()))
    else:
        channels_last_convs(m)
    dy = None
    F.set_backend("eager")
    try:
        dy = torch.randn_like(call(ref)[0])
        want, lib = gradients(ref, call, dy), gradients(plain, call, dy)
    finally:
        F.set_backend("fused")
    got = gradients(m, call, dy)
    assert got.keys() == want.keys()
    for k, w in want.items():
        assert got[k] is not None, k
        e, e0 = (((t[k].double() - w.double()).norm() / w.double().norm()).item() for t in (got, lib))
        assert e <= 3 * e0 + 2.0 ** -8, (k, e, e0)


def on_input(x, f):
    def call(m):
        p = next(m.parameters())
        ins = [t.to(p.dtype).detach().requires_grad_() for t in x]
        return f(m, *ins), ins
    return call


@pytest.mark.parametrize("arena", ["arena", "channels last"])
@pytest.mark.parametrize("cin,cout", [(64, 64), (64, 128)])
def test_unet_block(cin, cout, arena):
    m = randomised(ResBlock(cin, cout, 128, SDXLConfig(), torch.bfloat16, "cuda"))
    no_further_than_plain_bf16(m, on_input([nhwc(2, cin, 12, 10), torch.randn(2, 128, **KW)], lambda m, x, e: m(x, e)), arena)


class ConvThenBlock(nn.Module):
    def __init__(self, cin, cout):
        super().__init__()
        self.conv, self.blk = nn.Conv2d(32, cin, 3, padding=1, **KW), _Res(cin, cout, 32, KW)


@pytest.mark.parametrize("arena", ["arena", "channels last"])
@pytest.mark.parametrize("deferred", [False, True])
@pytest.mark.parametrize("cin,cout", [(64, 64), (64, 128)])
def test_autoencoder_block(cin, cout, deferred, arena):
    """``deferred``: the bias of the convolution in front is added by the block."""
    m = randomised(ConvThenBlock(cin, cout))
    seen = []

    def call(m, x):
        if not deferred:
            return m.blk(m.conv(x))
        seen.append(m.blk.fusable(x))
        return _run([m.conv, m.blk], x, lambda t: t)
    no_further_than_plain_bf16(m, on_input([nhwc(2, 32, 12, 10)], call), arena)
    assert not deferred or seen[-1]                 # (the last call is the folded one)


@pytest.mark.parametrize("arena", ["arena", "channels last"])
def test_autoencoder_encoder(arena):
    m = randomised(Encoder(VaeConfig(base=32, mult=(1, 2), layers_per_block=1), KW), seed=3)
    no_further_than_plain_bf16(m, on_input([nhwc(1, 3, 32, 24)], lambda m, x: m(x)), arena)
