"""Convolution with a trained weight in parameter order against fp64: channel counts around the 256-channel tiles, kernel sizes,
stride and dilation, gradients into a buffer and returned."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ci,co,k,stride,pad,dil", [(8, 16, 3, 1, 1, 1), (264, 24, 3, 1, 1, 1), (256, 8, 5, 2, 2, 1), (320, 64, 3, 1, 2, 2)])
@pytest.mark.parametrize("buffer", [True, False])
def test_trained_conv(ci, co, k, stride, pad, dil, buffer):
    g = torch.Generator(device="cuda").manual_seed(ci + co)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    conv = torch.nn.Conv2d(ci, co, k, stride, pad, dil, bias=False, dtype=torch.bfloat16, device="cuda")
    conv.weight.data = mk(co, ci, k, k) * (ci * k * k) ** -0.5
    if buffer:
        conv.weight.grad = mk(co, ci, k, k)
    start = conv.weight.grad.double() if buffer else 0
    x = mk(2, ci, 19, 22).to(memory_format=torch.channels_last).requires_grad_()
    y = F.conv_no_bias(conv, x)
    x64, w64 = x.detach().double().requires_grad_(), conv.weight.detach().double().requires_grad_()
    y64 = torch.nn.functional.conv2d(x64, w64, None, stride, pad, dil)
    dy = mk(*y.shape)
    y.backward(dy)
    dx, dw = torch.autograd.grad(y64, (x64, w64), dy.double())
    # one rounding to bf16 each (2^-9), the weight gradient's sum into the buffer a second one
    for a, b in ((y.detach(), y64.detach()), (x.grad, dx), (conv.weight.grad, dw + start)):
        assert ((a.double() - b).norm() / b.norm()).item() < 2 ** -7.5
