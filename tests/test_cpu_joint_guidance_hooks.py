"""Hooks anywhere in the UNet see one prediction per call: guidance is joined only when nobody listens."""
import pytest
import torch

from eridiffusion_b200.models import build_model
from eridiffusion_b200.sampling import pipelines as P


@pytest.mark.parametrize("where", ["conv_in", "down.0.0.conv1", "mid.1.blocks.0.attn1.to_qkv", "up.0.0", "every module"])
@pytest.mark.parametrize("pre", [False, True])
def test_hooks_see_the_callers_batch(where, pre):
    torch.manual_seed(0)
    unet = build_model("sdxl", device="cpu", dtype=torch.float32, block_channels=(32, 64, 64), transformer_depth=(0, 1, 1),
                       head_dim=16, context_dim=32, pooled_dim=16, addition_time_embed_dim=8).eval()
    sizes = []

    def hook(m, a, *y):
        if torch.is_tensor(a[0]) and a[0].dim() > 1:
            sizes.append(a[0].shape[0])
    if where == "every module":
        reg = torch.nn.modules.module.register_module_forward_pre_hook if pre else torch.nn.modules.module.register_module_forward_hook
        handle = reg(hook)
    else:
        m = unet.get_submodule(where)
        handle = (m.register_forward_pre_hook if pre else m.register_forward_hook)(hook)
    kw = dict(txt=torch.randn(1, 7, 32), pooled=torch.randn(1, 16), width=64, height=64, steps=1, seed=3, guidance_scale=3.0)
    try:
        P.UnifiedInferencePipeline(unet, P.ModelType.SDXL, device="cpu").generate(**kw)
    finally:
        handle.remove()
    assert sizes and set(sizes) == {1}
    assert unet.samples_independent()
