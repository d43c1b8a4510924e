"""The few-tile GEMM (K range split over a cluster) against fp64: edges of tiles and K steps, every split, operand majors,
row strides, LoRA K step and the epilogue family."""
import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


def _mk(g, *s):
    return torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)


def _close(y, r, K):
    # fp32 sums of bf16 products (K * 2^-24 at most) and one rounding of the result to bf16
    assert ((y.double() - r).norm() / r.norm()).item() < 2 ** -8 + K * 2 ** -24
    assert F.gemm_error_check() == 0


@pytest.mark.parametrize("splits", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(128, 128, 512), (129, 136, 520), (320, 512, 2048), (200, 1000, 584), (1024, 1280, 1288)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_products(M, N, K, splits, a_mn, b_mn):
    if a_mn:
        M, N = (M + 255) // 8 * 8, N + 128
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = _mk(g, K, M + 8)[:, :M] if a_mn else _mk(g, M, K + 8)[:, :K]       # rows of another stride
    b = _mk(g, K, N) if b_mn else _mk(g, N, K)
    out = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    y = F.gemm_native(a, b, out=out[:, :N], a_mn=a_mn, b_mn=b_mn, force_bn=-splits, alpha=0.5)
    a64, b64 = a.double(), b.double()
    r = 0.5 * (a64.t() if a_mn else a64) @ (b64 if b_mn else b64.t())
    _close(y, r, K)
    assert (out[:, N:] == 7).all()


@pytest.mark.parametrize("splits", [1, 4])
@pytest.mark.parametrize("act", [None, "gelu", "silu", "gelu_bwd"])
@pytest.mark.parametrize("rank", [0, 16, 64])
def test_epilogues(splits, act, rank):
    M, N, K, rows = 300, 264, 1000, 150
    g = torch.Generator(device="cuda").manual_seed(rank)
    a, b, bias, res, gate = _mk(g, M, K) * 0.05, _mk(g, N, K), _mk(g, N), _mk(g, M, N), _mk(g, 2, N)
    pre = _mk(g, M, N)
    kw, x64 = {}, a.double() @ b.double().t()
    if rank:
        h, lb = _mk(g, M, rank), _mk(g, N, rank)
        kw.update(lora_h=h, lora_b=lb)
        x64 = x64 + h.double() @ lb.double().t()
    x64 = x64 + bias.double()
    p_out = torch.empty_like(pre)
    if act in ("gelu", "silu"):
        kw.update(act=act, pre_out=p_out)
        y64 = torch.nn.functional.gelu(x64, approximate="tanh") if act == "gelu" else torch.nn.functional.silu(x64)
    elif act == "gelu_bwd":
        kw.update(act=act, pre_in=pre)
        p = pre.double().requires_grad_()
        (d,) = torch.autograd.grad(torch.nn.functional.gelu(p, approximate="tanh").sum(), p)
        y64 = x64 * d
    else:
        y64 = x64
    y64 = y64 * gate.double().repeat_interleave(rows, 0) + res.double()
    y = F.gemm_native(a, b, bias=bias, residual=res, gate=gate, rows_per_batch=rows, force_bn=-splits, **kw)
    # fast tanh / exponential of the activation: 2^-10 of its value
    assert ((y.double() - y64).norm() / y64.norm()).item() < 2 ** -8 + 2 ** -10
    if act in ("gelu", "silu"):
        assert ((p_out.double() - x64).norm() / x64.norm()).item() < 2 ** -8
    acc = res.clone()                                           # the result added into a buffer that is the residual too
    y2 = F.gemm_native(a, b, out=acc, residual=acc, force_bn=-splits)
    r2 = a.double() @ b.double().t() + res.double()
    _close(y2, r2, K)
