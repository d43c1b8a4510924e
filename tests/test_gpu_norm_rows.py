"""The CTA-per-row norm kernel against fp64, and against the row-per-warp kernel on both sides of the rule between them: widths
around each vectors-per-thread step, modulation, weights, bias, RMS and mean, an added gradient."""
import pytest
import torch

from eridiffusion_b200.ops import _native as N

pytestmark = pytest.mark.gpu


def _run(rows, D, rpb, rms, affine, mod, add, limit):
    lib = N.require()
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    x, dy, extra = mk(rows, D) + 2, mk(rows, D), mk(rows, D)
    B = (rows + rpb - 1) // rpb
    sc, sh, w, b = mk(B, D) * 0.3, mk(B, D), 1 + 0.1 * mk(D), mk(D)
    w = w.to(torch.bfloat16)
    y, dx = torch.empty_like(x), torch.empty_like(x)
    mean, rstd = torch.zeros(rows, device="cuda"), torch.zeros(rows, device="cuda")
    p = lambda t, on=True: t.data_ptr() if on else None  # noqa: E731
    lib.eri_norm_set_row_cta_rows(limit)
    try:
        N.check(lib.eri_norm_modulate_fwd_warp(p(x), p(sc, mod), p(sh, mod), p(w, affine), p(b, affine), p(y), p(mean), p(rstd), rows, D,
                                               rpb, D, 1e-6, int(rms), N.stream_ptr()), "fwd")
        N.check(lib.eri_norm_modulate_bwd_warp_add(p(dy), p(x), p(sc, mod), p(w, affine), p(mean), p(rstd), p(dx), p(extra, add), rows,
                                                   D, rpb, D, int(rms), N.stream_ptr()), "bwd")
    finally:
        lib.eri_norm_set_row_cta_rows(-1)
    x64 = x.double().requires_grad_()
    m = torch.zeros_like(x64[:, :1]) if rms else x64.mean(-1, keepdim=True)
    z = (x64 - m) * torch.rsqrt((x64 - m).pow(2).mean(-1, keepdim=True) + 1e-6)
    if affine:
        z = z * w.double() + b.double()
    if mod:
        idx = torch.arange(rows, device="cuda") // rpb
        z = z * (1 + sc.double()[idx]) + sh.double()[idx]
    (d64,) = torch.autograd.grad(z, x64, dy.double())
    return y, dx, z.detach(), d64 + (extra.double() if add else 0)


@pytest.mark.parametrize("limit", [0, 1 << 30])
@pytest.mark.parametrize("rows,D,rpb", [(1, 256, 1), (77, 1024, 77), (130, 1032, 65), (300, 2048, 100), (64, 2056, 64), (129, 3072, 43),
                                        (256, 3080, 256), (33, 4096, 11)])
@pytest.mark.parametrize("rms,affine,mod,add", [(False, False, True, False), (True, True, False, False), (False, True, True, True)])
def test_rows(rows, D, rpb, rms, affine, mod, add, limit):
    y, dx, y64, d64 = _run(rows, D, rpb, rms, affine, mod, add, limit)
    # fp32 statistics of bf16 rows, one rounding of the result to bf16 (2^-9)
    assert ((y.double() - y64).norm() / y64.norm()).item() < 2 ** -8
    assert ((dx.double() - d64).norm() / d64.norm()).item() < 2 ** -8
