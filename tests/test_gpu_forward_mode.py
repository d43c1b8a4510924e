"""Dual tensors are refused by every native op, with and without gradients recorded: none may come back without its tangent."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def mk(*s):
    return torch.randn(*s, device="cuda").to(torch.bfloat16)


X = (1, 256, 256)
lin = lambda: (mk(256, 256), None, None, None, None)  # noqa: E731
CASES = {
    "linear": (X, lambda t: F.linear(t, mk(256, 256))),
    "linear weight": ((256, 256), lambda t: F.linear(mk(*X), t)),
    "linear adapter": ((16, 256), lambda t: F.linear(mk(*X), mk(256, 256), lora=(t, mk(256, 16), 1.0))),
    "linear residual": (X, lambda t: F.linear(mk(*X), mk(256, 256), residual=t)),
    "linear gate": ((1, 256), lambda t: F.linear(mk(*X), mk(256, 256), residual=mk(*X), gate=t)),
    "linear_pair": (X, lambda t: F.linear_pair(t, lin(), mk(*X), lin())),
    "linear_pair residual": (X, lambda t: F.linear_pair(mk(*X), lin(), mk(*X), (*lin()[:3], t, mk(1, 256)))),
    "linear_pair gate": ((1, 256), lambda t: F.linear_pair(mk(*X), lin(), mk(*X), (*lin()[:3], mk(*X), t))),
    "small_linear": ((2, 64), lambda t: F.small_linear(t, mk(64, 64))),
    "norm": (X, lambda t: F.norm_modulate(t)),
    "norm scale": ((1, 256), lambda t: F.norm_modulate(mk(*X), scale=t)),
    "gate_residual": (X, lambda t: F.gate_residual(t, mk(*X))),
    "gelu": (X, F.gelu_tanh),
    "silu": (X, F.silu),
    "glu": (X, F.glu),
    "qknorm_rope": ((1, 64, 384), lambda t: F.qknorm_rope(t, None, None, None, None, 2)),
    "attention": ((1, 128, 2, 64), lambda t: F.attention(t, t, t)),
    "attention key mask": ((1, 1, 1, 128), lambda t: F.attention(*(mk(1, 128, 2, 64) for _ in range(3)), mask=t)),
    "attention query mask": ((1, 1, 128, 128), lambda t: F.attention(*(mk(1, 128, 2, 64) for _ in range(3)), mask=t)),
    "attention head 512": ((1, 128, 1, 512), lambda t: F.attention(t, t, t)),
    "attention_qkv": ((1, 128, 384), lambda t: F.attention_qkv(t, 2)),
    "attention_kv": ((1, 77, 256), lambda t: F.attention_kv(mk(1, 128, 128), t, 2)),
    "attention_qkv_rope": ((1, 128, 768), lambda t: F.attention_qkv_rope(t, mk(256), mk(256), *(torch.rand(128, 128, device="cuda") for _ in "cs"), 2)),
    "attention_qkv_rope weight": ((256,), lambda t: F.attention_qkv_rope(mk(1, 128, 768), t, mk(256),
                                                                         *(torch.rand(128, 128, device="cuda") for _ in "cs"), 2)),
    "group_norm": (X, lambda t: F.group_norm_silu(t, mk(256), mk(256))),
    "group_norm addend": ((256,), lambda t: F.group_norm_silu(mk(*X), mk(256), mk(256), pre_c=t)),
    "mse": (X, lambda t: F.mse_loss(t, mk(*X))),
}


@pytest.mark.parametrize("record", [True, False])
@pytest.mark.parametrize("name", CASES)
def test_refused(name, record):
    shape, fn = CASES[name]
    with fwAD.dual_level(), torch.set_grad_enabled(record):
        t = fwAD.make_dual(mk(*shape), torch.ones(shape, device="cuda", dtype=torch.bfloat16))
        with pytest.raises(NotImplementedError):
            fn(t)
    fn(mk(*shape))      # the same call on a plain tensor is answered


def test_split_tokens_keeps_the_tangent():
    with fwAD.dual_level():
        a, b = F.split_tokens(fwAD.make_dual(mk(*X), mk(*X)), 8)
        assert fwAD.unpack_dual(a).tangent is not None and fwAD.unpack_dual(b).tangent is not None
