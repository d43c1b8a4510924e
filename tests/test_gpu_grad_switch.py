"""With in-place accumulation switched off, no op writes into an existing gradient: every one is returned to autograd."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def mk(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


def conv(w, b):
    c = torch.nn.Conv2d(64, 64, 3, padding=1, device="cuda", dtype=torch.bfloat16)
    c.weight, c.bias = w, b
    x = mk(1, 64, 8, 8).contiguous(memory_format=torch.channels_last)
    return F.add_bias(x, F.conv_no_bias(c, x), b)


CASES = {
    "linear": ([(256, 128), (256,)], lambda w, b: F.linear(mk(1, 300, 128), w, b)),
    "adapter": ([(16, 128), (256, 16)], lambda a, b: F.linear(mk(1, 300, 128), mk(256, 128), lora=(a, b, 1.0))),
    "pair": ([(256, 128), (256,)], lambda w, b: F.linear_pair(mk(1, 300, 128), (w, b, None, None, None), mk(1, 300, 128),
                                                              (mk(256, 128), mk(256), None, None, None))[0]),
    "norm": ([(256,), (256,)], lambda w, b: F.norm_modulate(mk(1, 300, 256), weight=w, bias=b)),
    "group norm": ([(64,), (64,), (64,)], lambda w, b, c: F.group_norm_silu(mk(1, 200, 64), w, b, 8, pre_c=c)),
    "small linear": ([(256, 128)], lambda w: F.small_linear(mk(2, 128), w)),
    "convolution": ([(64, 64, 3, 3), (64,)], conv),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("on", [True, False])
def test_switch(monkeypatch, name, on):
    monkeypatch.setattr(F, "_ACCUM_INTO_GRAD", on)
    torch.manual_seed(0)
    shapes, fn = CASES[name]
    ps = [torch.nn.Parameter(mk(*s)) for s in shapes]
    torch.manual_seed(1)
    y = fn(*ps)
    dy = mk(*y.shape)
    y.backward(dy)
    want = [p.grad for p in ps]                      # no buffer: returned either way
    for p in ps:
        p.grad = torch.full_like(p, 2.0)
    versions = [p.grad._version for p in ps]
    torch.manual_seed(1)
    fn(*ps).backward(dy)
    for p, v, w in zip(ps, versions, want):
        # autograd's own addition counts as a change of the buffer, a kernel's write through its pointer does not
        assert on or p.grad._version > v
        assert (p.grad.double() - 2 - w.double()).abs().max() <= 2.0 ** -7 * (2 + w.abs().max().item())
