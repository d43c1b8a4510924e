"""Probabilities of the per-query-mask attention keep fp32's mantissa through the second product: results that cancel to 2^-13
of their terms show any bit that is lost before it."""
import math

import pytest
import torch

from eridiffusion_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
def test_cancelling_values(D):
    H = 48
    g = torch.Generator().manual_seed(D)
    delta = (torch.rand(H, generator=g) * 0.6 + 0.02).to(torch.bfloat16)
    grid = 1 + torch.arange(128, dtype=torch.float64) / 128            # the bf16 numbers of [1, 2)
    v = torch.zeros(1, 2, H, D, dtype=torch.float64)
    for h in range(H):
        # out = (a - p b) / (1 + p) with a - p b nearly zero, for D pairs (a, b)
        diff = grid[:, None] / 2 - math.exp(-float(delta[h])) * grid[None] / 2
        i = diff.abs().flatten().argsort()[:D]
        v[0, 0, h], v[0, 1, h] = grid[i // 128] / 2, -grid[i % 128] / 2
    mask = torch.zeros(1, H, 16, 2)
    mask[0, :, :, 1] = -delta.float()[:, None]
    q, k = torch.zeros(1, 16, H, D), torch.ones(1, 2, H, D)
    q, k, vb, mask = (t.to("cuda", torch.bfloat16) for t in (q, k, v, mask))
    o = F.attention(q, k, vb, mask=mask).double().cpu()
    p = torch.exp(-delta.double())
    want = (v[0, 0] + p[:, None] * v[0, 1]) / (1 + p[:, None])
    near = want.abs() < 2.0 ** -12         # where the result's own rounding is below 2^-21
    assert torch.equal(vb.double().cpu(), v) and near.sum() > 100
    # the exponential is good to 2^-22; two bf16 terms of a probability leave 2^-18
    assert ((o[0] - want[None]).abs() * near).max().item() < 2.0 ** -20.5
