"""Performance cases: what a user of the framework has it do, each through the entry points that the
training and sampling commands call.

    train_mmdit   ``Trainer.train_step`` on the FLUX-style / Qwen-Image-style / tiny MMDiT
    train_video   ``Trainer.train_step`` on the LTX-style video DiT
    train_unet    ``Trainer.train_step`` on the SDXL UNet
    sample_mmdit  ``generate_flow``: Euler sampling of latents from the FLUX-style MMDiT
    sample_unet   ``UnifiedInferencePipeline.generate``: classifier-free guided sampling from the SDXL UNet
    vae           ``AutoencoderKL.encode`` / ``decode``
    text          T5-style and CLIP-style prompt encoding
    optimizer     gradient norm, ``AdamW8bit.step`` and the weight average on a flat parameter arena

Widths, head counts, latent layouts and text lengths are those of ``models/``, ``data.synthetic_batch`` and
``bench.py``. The transformer stacks keep their full width and lose depth (every block of a stack does the
same work), so that a case is prepared quickly. Weights are random-init, inputs N(0, 1) like the latents and
embeddings that the models train on.
"""
from __future__ import annotations

import math

import torch

from eridiffusion_b200.adapters import AdapterConfig
from eridiffusion_b200.models import build_model
from eridiffusion_b200.models.sdxl_unet import sdxl_forward
from eridiffusion_b200.ops import functional as F
from eridiffusion_b200.optim import EMA, ParamArena
from eridiffusion_b200.optim.adamw8bit import AdamW8bit
from eridiffusion_b200.sampling import generate_flow
from eridiffusion_b200.sampling.pipelines import ModelType, UnifiedInferencePipeline
from eridiffusion_b200.train.trainer import Trainer, TrainerConfig, default_forward, ltx_forward

BF16 = torch.bfloat16
DEV = "cuda"


def listed():
    return [
        # The smallest training job: the tiny MMDiT that setups are tried out with. Latency and launches count.
        dict(name="tiny lora step", kind="train_mmdit", family="tiny_mmdit", mode="lora", rank=16, batch=2, height=256,
             width=256, text=64, double=2, single=2, accum=1),
        # Low-resolution LoRA training, gradients accumulated over four micro-batches: few tokens per launch.
        dict(name="flux lora 256px", kind="train_mmdit", family="flux", mode="lora", rank=16, batch=1, height=256,
             width=256, text=128, double=1, single=2, accum=4),
        # The headline configuration of bench.py: LoRA r16 at 1024 x 1024 with 512 text tokens.
        dict(name="flux lora 1024px", kind="train_mmdit", family="flux", mode="lora", rank=16, batch=1, height=1024,
             width=1024, text=512, double=2, single=4, accum=1),
        # An aspect-ratio bucket: 832 x 1216 with a text length that no tile divides, batch 2, rank 32.
        dict(name="flux lora 832x1216 b2", kind="train_mmdit", family="flux", mode="lora", rank=32, batch=2, height=1216,
             width=832, text=333, double=1, single=2, accum=2),
        # Full fine-tune of the dual-stream stack: weight gradients of every layer, 8-bit AdamW on all parameters.
        dict(name="qwen full 1024px", kind="train_mmdit", family="qwen_image", mode="full", rank=0, batch=1, height=1024,
             width=1024, text=256, double=2, single=0, accum=2),
        # Video LoRA on the 33-frame clip of 19008 tokens: self-attention over a long sequence is the largest part.
        dict(name="ltx lora 33 frames", kind="train_video", mode="lora", rank=16, batch=1, frames=33, h=24, w=24, text=256,
             depth=1, accum=2),
        # UNet full fine-tune at 1024 x 1024: convolutions, GroupNorm, self- and cross-attention at head size 64.
        dict(name="sdxl full 1024px", kind="train_unet", mode="full", rank=0, batch=1, height=1024, width=1024, depth1=2,
             depth2=10, accum=2),
        # Validation image during training: four Euler steps at 512 x 512.
        dict(name="flux sample 512px", kind="sample_mmdit", batch=1, height=512, width=512, text=512, double=2, single=4,
             steps=4),
        # Classifier-free guided UNet sampling: two denoiser calls per step at batch 1.
        dict(name="sdxl sample 1024px", kind="sample_unet", batch=1, height=1024, width=1024, depth1=2, depth2=10, steps=2,
             sampler="euler"),
        # Latents to an image at the end of sampling.
        dict(name="vae decode 1024px", kind="vae", family="vae_sdxl", direction="decode", batch=1, height=1024, width=1024),
        # One caption through the T5-style encoder when the embedding cache is built.
        dict(name="t5 encode 256", kind="text", family="t5_encoder", batch=1, tokens=256, layers=8),
        # Optimizer update of a full fine-tune (the arena of a few large blocks) with the weight average on.
        dict(name="adamw8bit 400M ema", kind="optimizer", numel=400_000_000, ema=True),
    ]


# ------------------------------------------------------------------------------------------- drawing cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi, step):
    return max(lo // step, _log(rng, lo, hi) // step) * step


def draw(rng):
    kind = rng.choice(["train_mmdit", "train_mmdit", "train_mmdit", "train_video", "train_unet", "sample_mmdit",
                       "sample_unet", "vae", "text", "optimizer"])
    if kind == "train_mmdit":
        family = rng.choice(["flux", "flux", "qwen_image", "tiny_mmdit"])
        h, w = _side(rng, 256, 1280, 16), _side(rng, 256, 1280, 16)
        text = _log(rng, 64, 512)
        tokens = (h // 16) * (w // 16) + text
        mode = "full" if family == "qwen_image" and rng.random() < 0.7 else "lora"
        return dict(kind=kind, family=family, mode=mode, rank=rng.choice([16, 32, 64]) if mode == "lora" else 0,
                    batch=rng.randint(1, max(1, min(4, 9000 // tokens))), height=h, width=w, text=text,
                    double=rng.randint(1, 2), single=0 if family == "qwen_image" else rng.randint(1, 3),
                    accum=rng.randint(1, 4))
    if kind == "train_video":
        return dict(kind=kind, mode="lora", rank=rng.choice([16, 32, 64]), batch=1, frames=_log(rng, 1, 32),
                    h=_log(rng, 8, 24), w=_log(rng, 8, 24), text=_log(rng, 64, 512), depth=1, accum=rng.randint(1, 4))
    if kind == "train_unet":
        h, w = _side(rng, 512, 1280, 64), _side(rng, 512, 1280, 64)
        mode = rng.choice(["full", "lora"])
        return dict(kind=kind, mode=mode, rank=16 if mode == "lora" else 0,
                    batch=rng.randint(1, max(1, (1024 * 1024) // (h * w))), height=min(h, 1024 * 1024 // w // 64 * 64),
                    width=w, depth1=rng.randint(1, 2), depth2=rng.randint(2, 10), accum=rng.randint(1, 4))
    if kind == "sample_mmdit":
        h, w = _side(rng, 256, 1024, 16), _side(rng, 256, 1024, 16)
        return dict(kind=kind, batch=1, height=h, width=w, text=_log(rng, 64, 512), double=rng.randint(1, 2),
                    single=rng.randint(1, 4), steps=rng.randint(1, min(8, 20000 // ((h // 16) * (w // 16) + 512))))
    if kind == "sample_unet":
        return dict(kind=kind, batch=1, height=_side(rng, 512, 1024, 64), width=_side(rng, 512, 1024, 64),
                    depth1=rng.randint(1, 2), depth2=rng.randint(2, 10), steps=rng.randint(1, 2),
                    sampler=rng.choice(["euler", "dpmpp_2m"]))
    if kind == "vae":
        return dict(kind=kind, family=rng.choice(["vae_sdxl", "vae_flux"]), direction=rng.choice(["encode", "decode"]),
                    batch=1, height=_side(rng, 256, 1024, 8), width=_side(rng, 256, 1024, 8))
    if kind == "text":
        if rng.random() < 0.3:
            return dict(kind=kind, family="clip_l", batch=rng.randint(1, 8), tokens=77, layers=12)
        return dict(kind=kind, family="t5_encoder", batch=rng.randint(1, 4), tokens=_log(rng, 64, 512),
                    layers=rng.randint(4, 8))
    return dict(kind=kind, numel=_log(rng, 1 << 20, 400_000_000), ema=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------- models and inputs
def _model(c, device):
    kind = c["kind"]
    if kind in ("train_mmdit", "sample_mmdit"):
        family = c.get("family", "flux")
        return build_model(family, dtype=BF16, device=device, depth_double=c["double"], depth_single=c["single"])
    if kind == "train_video":
        return build_model("ltx_video", dtype=BF16, device=device, depth=c["depth"])
    if kind in ("train_unet", "sample_unet"):
        return build_model("sdxl", dtype=BF16, device=device, transformer_depth=(0, c["depth1"], c["depth2"]))
    if kind == "vae":
        return build_model(c["family"], dtype=BF16, device=device)
    return build_model(c["family"], dtype=BF16, device=device, layers=c["layers"])


def _unit_gain(model):
    """Convolution weights that keep the variance of their input, as trained ones roughly do: with PyTorch's default
    (a third of it) every normalisation that follows also scales the rounding of the layers before it up."""
    with torch.no_grad():
        for m in model.modules():
            if isinstance(m, torch.nn.Conv2d):
                m.weight.mul_(3 ** 0.5)


def _size_ids(c, device):
    h, w = c["height"], c["width"]
    return torch.tensor([[h, w, 0, 0, h, w]] * c["batch"], dtype=torch.float32, device=device)


def _batch(c, mk, device):
    """One micro-batch of cached latents and embeddings; ``mk(*shape)`` makes an N(0, 1) bf16 tensor."""
    B = c["batch"]
    if c["kind"] == "train_video":
        return {"latents": mk(B, 128, c["frames"] * c["h"] * c["w"], 1), "txt": mk(B, c["text"], 4096),
                "grid_fhw": (c["frames"], c["h"], c["w"])}
    h, w = c["height"] // 8, c["width"] // 8
    if c["kind"] == "train_unet":
        return {"latents": mk(B, 4, h, w), "txt": mk(B, 77, 2048), "pooled": mk(B, 1280), "time_ids": _size_ids(c, device)}
    width, pooled = {"flux": (4096, 768), "qwen_image": (3584, 0), "tiny_mmdit": (128, 64)}[c["family"]]
    b = {"latents": mk(B, 16, h, w), "txt": mk(B, c["text"], width), "grid_hw": (h // 2, w // 2)}
    if pooled:
        b["pooled"] = mk(B, pooled)
    return b


_FORWARD = {"train_mmdit": default_forward, "train_video": ltx_forward, "train_unet": sdxl_forward}


def prepare(case, seed):
    c = dict(case)
    g = torch.Generator(device=DEV).manual_seed(seed)
    torch.manual_seed(seed)

    def mk(*s):
        return torch.randn(*s, device=DEV, generator=g, dtype=torch.float32).to(BF16)

    kind = c["kind"]
    if kind == "optimizer":
        p = torch.nn.Parameter(mk(c["numel"]).mul_(0.02))
        arena = ParamArena([p])
        # gradients of a batch: a few decades between the layers' magnitudes
        arena.grad[:c["numel"]].copy_(mk(c["numel"])).mul_(1e-3)
        arena.grad[: c["numel"] // 2].mul_(0.1)
        opt = AdamW8bit(arena, lr=1e-5, seed=seed)
        return dict(c=c, arena=arena, opt=opt, ema=EMA(arena, 0.999) if c["ema"] else None, sumsq=None)
    model = _model(c, DEV)
    if kind in ("train_unet", "vae"):
        _unit_gain(model)
    if kind.startswith("train_"):
        unet = kind == "train_unet"
        # adapters that are past their zero start, as in every step but the first; several trainers live in one
        # process here, so the collector is left alone (``gc_freeze_after`` is for one trainer per process)
        adapter = AdapterConfig(rank=c["rank"], alpha=c["rank"], init="nonzero") if c["mode"] == "lora" else None
        cfg = TrainerConfig(mode=c["mode"], adapter=adapter, objective="eps" if unet else "flow",
                            guidance=3.5 if c.get("family") == "flux" else None, optimizer="adamw8bit", lr=1e-4 if adapter else 1e-5,
                            grad_accum=c["accum"], patch=2 if kind == "train_mmdit" else 1, seed=seed, gc_freeze_after=0)
        tr = Trainer(model, cfg, forward_fn=_FORWARD[kind])
        return dict(c=c, trainer=tr, batch=_batch(c, mk, DEV))
    model.eval().requires_grad_(False)
    B = c["batch"]
    if kind == "sample_mmdit":
        return dict(c=c, model=model, txt=mk(B, c["text"], 4096), pooled=mk(B, 768), seed=seed)
    if kind == "sample_unet":
        pipe = UnifiedInferencePipeline(model, ModelType.SDXL)
        return dict(c=c, pipe=pipe, txt=mk(B, 77, 2048), pooled=mk(B, 1280), neg_txt=mk(B, 77, 2048),
                    neg_pooled=mk(B, 1280), seed=seed)
    if kind == "vae":
        x = mk(B, 3, c["height"], c["width"]).clamp_(-1, 1) if c["direction"] == "encode" else \
            mk(B, model.cfg.latent_channels, c["height"] // 8, c["width"] // 8).mul_(model.cfg.scaling_factor)
        return dict(c=c, vae=model, x=x)
    ids = torch.randint(0, model.cfg.vocab_size - 1, (B, c["tokens"]), device=DEV, generator=g)
    if c["family"] == "clip_l":
        with torch.no_grad():
            model.position_embedding.copy_(mk(c["tokens"], model.cfg.hidden).mul_(0.01))
            model.token_embedding.weight.mul_(0.02)
        ids[:, -1] = model.cfg.eos_token_id
        return dict(c=c, enc=model, ids=ids)
    with torch.no_grad():       # T5's scores are unscaled: its query weights start d_head ** -0.5 smaller
        for ly in model.layers:
            ly.qkv.weight[: model.cfg.heads * model.cfg.head_dim].mul_(model.cfg.head_dim ** -0.5)
    lengths = torch.randint(max(1, c["tokens"] // 4), c["tokens"] + 1, (B, 1), device=DEV, generator=g)
    return dict(c=c, enc=model, ids=ids, mask=torch.arange(c["tokens"], device=DEV)[None] < lengths)


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind.startswith("train_"):
        tr = state["trainer"]
        loss = tr.train_step(state["batch"])
        return {"loss": loss, "params": tr.arena.data, "grads": tr.arena.grad, "m_absmax": tr.optimizer.m_absmax,
                "v_absmax": tr.optimizer.v_absmax}
    if kind == "optimizer":
        opt, arena = state["opt"], state["arena"]
        state["sumsq"] = F.sumsq(arena.grad, state["sumsq"])
        opt.step(grad_sumsq=state["sumsq"], max_grad_norm=1.0)
        out = {"params": arena.data, "m_q": opt.m_q, "v_q": opt.v_q, "m_absmax": opt.m_absmax, "v_absmax": opt.v_absmax}
        if state["ema"] is not None:
            state["ema"].update()
            out["ema"] = state["ema"].shadow
        return out
    if kind == "sample_mmdit":
        return generate_flow(state["model"], state["txt"], state["pooled"], c["height"], c["width"], steps=c["steps"],
                             seed=state["seed"])
    if kind == "sample_unet":
        # guidance 2: the two predictions of a random-init UNet hardly differ, a larger scale multiplies their rounding
        return state["pipe"].generate(width=c["width"], height=c["height"], steps=c["steps"], seed=state["seed"],
                                      guidance_scale=2.0, txt=state["txt"], pooled=state["pooled"], neg_txt=state["neg_txt"],
                                      neg_pooled=state["neg_pooled"], sampler=c["sampler"])
    with torch.no_grad():
        if kind == "vae":
            return state["vae"].encode(state["x"], sample=False) if c["direction"] == "encode" else \
                state["vae"].decode(state["x"])
        if c["family"] == "clip_l":
            return state["enc"](state["ids"])
        return state["enc"](state["ids"], state["mask"])


# ------------------------------------------------------------------------------------------- work and tolerance
def _denoiser_calls(c):
    if c["kind"] == "sample_mmdit":
        return c["steps"]
    return 2 * c["steps"]       # classifier-free guidance calls the UNet twice per step


def work(case):
    """Operations of the path's matrix products, attention and convolutions (forward, input gradients and, where
    weights train, weight gradients; an adapter's own are left out), counted on a shape-only copy of the model. Bytes:
    weights once, inputs once, outputs (and the trained state) once."""
    c = dict(case)
    kind = c["kind"]
    if kind == "optimizer":
        n = c["numel"]
        per = 2 + (2 + 1 + 1) * 2 + 8 * 2 / 256 + (8 if c["ema"] else 0)   # gradient; parameter and codes both ways
        return {"bytes": per * n, "flops": 30 * n}
    from torch.utils.flop_counter import FlopCounterMode

    def mk(*s):
        return torch.empty(*s, device="meta", dtype=BF16)

    model = _model(c, "meta")
    n_params = sum(p.numel() for p in model.parameters())
    B = c["batch"]
    counter = FlopCounterMode(display=False)
    if kind.startswith("train_"):
        model.requires_grad_(c["mode"] == "full")
        b = _batch(c, mk, "meta")
        D = {"train_mmdit": 64, "train_video": 128, "train_unet": 4}[kind]
        x = mk(B, b["latents"].numel() // (B * D), D)
        cfg = TrainerConfig(guidance=3.5 if c.get("family") == "flux" else None)
        with counter:
            y = _FORWARD[kind](model, x.requires_grad_(c["mode"] == "lora"), torch.empty(B, device="meta"), b, cfg)
            y.sum().backward()
        flops = counter.get_total_flops()
        # full: parameter and gradient read and written, two one-byte moments read and written every accum-th pass
        state = n_params * (4 + 10 / c["accum"]) if c["mode"] == "full" else 0
        return {"bytes": 2 * n_params + state + 2 * (3 * x.numel() + b["txt"].numel()), "flops": flops}
    with torch.no_grad(), counter:
        if kind == "sample_mmdit":
            h, w = c["height"] // 16, c["width"] // 16
            x = mk(B, h * w, 64)
            y = model(x, mk(B, c["text"], 4096), torch.empty(B, device="meta"), mk(B, 768), grid_hw=(h, w))
        elif kind == "sample_unet":
            x = mk(B, 4, c["height"] // 8, c["width"] // 8)
            y = model(x, torch.empty(B, device="meta"), mk(B, 77, 2048), mk(B, 1280), _size_ids(c, "meta"))
        elif kind == "vae" and c["direction"] == "encode":
            x = mk(B, 3, c["height"], c["width"])
            y = model.encode(x, sample=False)
        elif kind == "vae":
            x = mk(B, model.cfg.latent_channels, c["height"] // 8, c["width"] // 8)
            y = model.decode(x)
        else:
            x = torch.zeros(B, c["tokens"], dtype=torch.long, device="meta")
            y = model(x)[0] if c["family"] == "clip_l" else model(x)
    if kind == "vae":       # the other half of the autoencoder is not read
        half = model.encoder if c["direction"] == "encode" else model.decoder
        n_params = sum(p.numel() for p in half.parameters())
    calls = _denoiser_calls(c) if kind.startswith("sample_") else 1
    return {"bytes": calls * (2 * n_params + 2 * (x.numel() + y.numel())), "flops": calls * counter.get_total_flops()}


def tolerance(case):
    kind = case["kind"]
    if kind == "optimizer":
        # fp32 arithmetic on both sides, one rounding to bf16 (stochastic, from a counter stream): 2^-8 on the few
        # parameters that land on the other side; a code moves by one where the value sits on a boundary
        return {"rel": 1e-3, "max": 2e-2, "differ": 2e-3}
    if kind.startswith("train_"):
        # every activation and gradient is rounded to bf16 between layers; the largest difference sits in gradients
        # that are small sums of many terms
        return {"rel": 2e-2, "max": 0.9 if kind == "train_unet" else 0.6}
    return {"rel": 2e-2, "max": 0.3}
