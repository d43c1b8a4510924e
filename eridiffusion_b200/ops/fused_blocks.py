"""Block-level fusions: the FLUX single-stream block as one autograd node.

The block computes ``x + gate * linear2(cat(attn(qkv), gelu(mlp)))`` where ``qkv`` and ``mlp`` are
column ranges of one projection ``linear1``. Written with separate ops this needs a split, an
activation pass and a concatenation in forward and zero-fill / copy / add passes for the slice
gradients in backward. Here the column-split epilogue of the GEMM writes the qkv columns and
``gelu(mlp)`` straight to where the next op reads them (the activation output lands inside the
concatenated buffer), and backward produces the gradient of the wide projection output in place:
the attention-gradient columns come from the QK-norm/RoPE backward with a row stride, the MLP
columns from linear2's input-gradient GEMM with the GELU-derivative epilogue.

Reference block: single blocks of src/models/flux_model_complete.rs:830-956 (linear1
[3D+4D, D], linear2 [D, D+4D], QK-norm, 3-way modulation).
"""
from __future__ import annotations

import torch

from . import _native as N
from . import flash_attn as FA
from . import functional as F


# GELU of the MLP half in the first linear's epilogue (forward) / its derivative in the second linear's
# input-gradient epilogue (backward), or as row passes of their own. Measured with eight epilogue warps at
# [4608 x 12288 x 3072]: storing activation + pre-activation from the epilogue 296 us against 244 + 43 us, the
# derivative in the epilogue 280 us against 250 + 55 us: the forward pass stays separate, the backward is fused.
_ACT_FWD_IN_EPILOGUE = __import__("os").environ.get("ERI_B200_SS_ACT_EPILOGUE", "0") == "1"
_ACT_BWD_IN_EPILOGUE = __import__("os").environ.get("ERI_B200_SS_ACT_BWD_EPILOGUE", "1") == "1"


def single_stream_supported(xm, gate, lin1, lin2, heads) -> bool:
    if not (xm.is_cuda and xm.dtype == torch.bfloat16 and F.get_backend() == "fused"):
        return False
    if F._GEMM_NATIVE != "native" or F._ATTN_NATIVE != "native" or not FA.has_backward():
        return False
    B, L, D = xm.shape
    if B * L < 128 or L < 128 or D // heads not in (64, 128) or D % 256 or gate.requires_grad:
        return False
    for lin in (lin1, lin2):
        ad = getattr(lin, "adapter", None)
        if type(lin).__name__ != "Linear":
            return False
        if ad is not None and not (getattr(ad, "kind", "") == "lora" and ad.rank in (16, 32, 64)
                                   and not (ad.dropout > 0 and ad.training)):
            return False
    return True


def single_stream(xm, x, gate, lin1, lin2, q_scale, k_scale, cos, sin, heads):
    """xm: modulated/normalised input [B, L, D]; x: residual stream; gate [B, D]."""
    def lora(lin):
        ad = getattr(lin, "adapter", None)
        return (None, None, 1.0) if ad is None else (ad.lora_A, ad.lora_B, float(ad.scale))
    a1, bb1, s1 = lora(lin1)
    a2, bb2, s2 = lora(lin2)
    cosf = None if cos is None else cos.float().contiguous()
    sinf = None if sin is None else sin.float().contiguous()
    return N.ops().single_stream(xm, x, gate, lin1.weight, lin1.bias, lin2.weight, lin2.bias, a1, bb1, s1, a2, bb2, s2,
                                 q_scale, k_scale, cosf, sinf, heads, F._flags(), _ACT_FWD_IN_EPILOGUE, _ACT_BWD_IN_EPILOGUE)
