"""Classifier-free guidance with both predictions in one call gives what two calls give, and calls that cannot be joined
are still answered by two."""
import pytest
import torch

from eridiffusion_b200.models import build_model
from eridiffusion_b200.sampling import pipelines as P


@pytest.mark.parametrize("batch,sampler,neg_len,joint", [(1, "euler", 7, True), (2, "dpmpp_2m", 7, True), (1, "euler_a", None, True),
                                                         (1, "euler", 5, False), (1, "hooked", 7, False)])
def test_joint_guidance(monkeypatch, batch, sampler, neg_len, joint):
    torch.manual_seed(0)
    unet = build_model("sdxl", device="cpu", dtype=torch.float32, block_channels=(32, 64, 64), transformer_depth=(0, 1, 1),
                       head_dim=16, context_dim=32, pooled_dim=16, addition_time_embed_dim=8).eval()
    sizes = []
    fwd = unet.forward
    unet.forward = lambda x, *a, **k: (sizes.append(x.shape[0]), fwd(x, *a, **k))[1]
    if sampler == "hooked":
        unet.register_forward_pre_hook(lambda m, a: None)
        sampler = "euler"
    pipe = P.UnifiedInferencePipeline(unet, P.ModelType.SDXL, device="cpu")
    kw = dict(txt=torch.randn(batch, 7, 32), pooled=torch.randn(batch, 16), width=64, height=64, steps=2, seed=3, guidance_scale=3.0,
              sampler=sampler)
    if neg_len is not None:
        kw.update(neg_txt=torch.randn(batch, neg_len, 32), neg_pooled=torch.randn(batch, 16))
    a = pipe.generate(**kw)
    assert set(sizes) == {2 * batch if joint else batch}
    monkeypatch.setattr(P, "_JOINT_GUIDANCE_PIXELS", 0)
    sizes.clear()
    b = pipe.generate(**kw)
    assert set(sizes) == {batch}
    # fp32 products of another row count: some 1e-6 of rounding, passed through two steps
    torch.testing.assert_close(a, b, rtol=1e-3, atol=1e-3)
