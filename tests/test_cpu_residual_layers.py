"""Layers whose residual sum moved into their call: a replaced layer needs no residual argument, a hook sees the layer's own
output, and both give what the plain layer gives."""
import pytest
import torch
import torch.nn as nn

from eridiffusion_b200.models.sdxl_unet import SDXLConfig, Transformer2D
from eridiffusion_b200.models.text_encoders import T5Config, _T5Layer


def t5():
    m = _T5Layer(T5Config(hidden=32, heads=2, head_dim=16, ff=48), dict(dtype=torch.float32))
    return m, (torch.randn(2, 7, 32), torch.zeros(2, 2, 7, 7))


def transformer():
    m = Transformer2D(32, 1, SDXLConfig(head_dim=16, context_dim=24), torch.float32, None)
    return m, (torch.randn(2, 32, 4, 4), torch.randn(2, 5, 24))


@pytest.mark.parametrize("make,name", [(t5, "o"), (t5, "wo"), (transformer, "proj_out")])
def test_replaced_or_hooked(make, name):
    torch.manual_seed(0)
    m, args = make()
    want = m(*args)
    lin, own = getattr(m, name), []
    handle = lin.register_forward_hook(lambda _, a, y: own.append((a[0], y)))
    torch.testing.assert_close(m(*args), want)
    torch.testing.assert_close(own[0][1], nn.functional.linear(own[0][0], lin.weight, lin.bias))
    handle.remove()
    other = nn.Linear(lin.in_features, lin.out_features, bias=lin.bias is not None)
    other.load_state_dict(lin.state_dict())
    setattr(m, name, other)
    torch.testing.assert_close(m(*args), want)
