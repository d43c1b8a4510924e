"""Public op surface. CUDA bf16 tensors run the hand-written sm_100a kernels (through autograd
nodes of the native op layer, ``csrc/torch``); everything else runs the PyTorch statements in
``reference``. ``set_backend("eager")`` forces the PyTorch path on CUDA too — that is the
library baseline the fused path is measured against.
"""
from __future__ import annotations

import math
import os

import torch

from . import _native as N
from . import reference as R

_BACKEND = os.environ.get("ERI_B200_BACKEND", "fused")  # "fused" | "eager"
_GEMM_NATIVE = os.environ.get("ERI_B200_GEMM", "native")  # "native" | "library"
_ATTN_NATIVE = os.environ.get("ERI_B200_ATTN", "native")  # "native" | "library"
_GEMM_PAIR = os.environ.get("ERI_B200_GEMM2", "1") == "1"  # two-CTA tiles for large problems
_PAIR_MIN_TILES = int(os.environ.get("ERI_B200_PAIR_MIN_TILES", "36"))  # at most this many 256 x 256 tiles: one-CTA kernel
_GATHER_JOIN = os.environ.get("ERI_B200_GATHER_JOIN", "0") == "1"  # copy clusters compute tiles after copying
_GATHER_PAIR = os.environ.get("ERI_B200_GATHER_PAIR", "1") == "1"  # gather-fused GEMMs on the two-CTA kernel
_GATHER_LOCAL = os.environ.get("ERI_B200_GATHER_LOCAL", "1") == "1"  # own slab read in place, not copied
_SCATTER_PAIR = os.environ.get("ERI_B200_SCATTER_PAIR", "1") == "1"  # peer-scatter epilogue on the two-CTA kernel
_WGRAD_NATIVE = os.environ.get("ERI_B200_WGRAD", "native") == "native"  # weight gradients on tcgen05 (else torch.mm)
_RANK_STREAM = os.environ.get("ERI_B200_RANK_STREAM", "1") == "1"  # streaming kernel for [M,K] x [r,K]^T
# Launch the LoRA-fused GEMM as a programmatic dependent of the down-projection kernel that precedes
# it on the stream: its main K loop overlaps that kernel and only the rank-r step waits for it.
_PDL = os.environ.get("ERI_B200_PDL", "1") == "1"


def _pdl_ok() -> bool:
    # the overlap is only sound when the down-projection is the launch right before the GEMM;
    # deterministic mode makes torch.empty launch a fill kernel in between
    return _PDL and not torch.are_deterministic_algorithms_enabled()


def set_backend(name: str) -> None:
    global _BACKEND
    if name not in ("fused", "eager"):
        raise ValueError(name)
    _BACKEND = name


def get_backend() -> str:
    return _BACKEND


def set_gemm_impl(name: str) -> None:
    global _GEMM_NATIVE
    _GEMM_NATIVE = name


def set_attention_impl(name: str) -> None:
    global _ATTN_NATIVE
    _ATTN_NATIVE = name


def _native_ok(*ts) -> bool:
    if _BACKEND != "fused":
        return False
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda or t.dtype != torch.bfloat16:
            return False
    N.require()
    return True


def _c(t):
    return None if t is None else (t if t.is_contiguous() else t.contiguous())


def _mod_view(t, D):
    """A [B, D] modulation tensor whose rows may be strided (a chunk of a wider tensor)."""
    if t is None:
        return None, 0
    assert t.dim() == 2 and t.shape[1] == D
    if t.stride(1) != 1 or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t, t.stride(0)


# ---------------------------------------------------------------------------- norm + modulation
def norm_modulate_skip(x, scale=None, shift=None, weight=None, bias=None, eps=1e-6, rms=False):
    """``(norm_modulate(x, ...), x)``: the second value is x for the residual branch around the norm. On the
    native path the gradients of both branches are summed inside the norm's backward kernel."""
    if _NORM_SKIP and _native_ok(x, scale, shift, weight, bias) and x.dim() == 3 and x.shape[-1] % 8 == 0 \
            and torch.is_grad_enabled() and x.requires_grad:
        return N.ops().norm_modulate(x, scale, shift, weight, bias, eps, rms, True, _ACCUM_INTO_GRAD)
    return norm_modulate(x, scale, shift, weight, bias, eps, rms), x


# Off by default: the FLUX LoRA step measured 190.0 / 192.8 ms with it and 190.5 / 191.0 ms without (alternating runs).
_NORM_SKIP = os.environ.get("ERI_B200_NORM_SKIP", "0") == "1"


def norm_modulate(x, scale=None, shift=None, weight=None, bias=None, eps=1e-6, rms=False):
    if _native_ok(x, scale, shift, weight, bias) and x.dim() == 3 and x.shape[-1] % 8 == 0 \
            and x.shape[-1] <= 8192:
        return N.ops().norm_modulate(x, scale, shift, weight, bias, eps, rms, False, _ACCUM_INTO_GRAD)[0]
    return R.norm_modulate(x, scale, shift, weight, bias, eps, rms)


# ---------------------------------------------------------------------------- QK-norm + RoPE
def qknorm_rope(qkv, q_scale, k_scale, cos, sin, num_heads, eps=1e-6):
    """qkv [B, L, 3*H*Dh] -> q, k, v [B, L, H, Dh] (norm + rotary on q, k)."""
    return qknorm_rope_joint([(qkv, q_scale, k_scale)], cos, sin, num_heads, eps)


def qknorm_rope_joint(streams, cos, sin, num_heads, eps=1e-6):
    """streams: list of (qkv [B, L_i, 3*H*Dh], q_scale [Dh] | None, k_scale [Dh] | None).
    Returns joint q, k, v [B, sum L_i, H, Dh]; cos/sin [sum L_i, Dh/2] or None."""
    W = streams[0][0].shape[-1]
    Dh = W // (3 * num_heads)
    tens = [t for s in streams for t in s]
    if _native_ok(*tens) and Dh in (64, 128) and (cos is None or cos.is_cuda):
        cosf = None if cos is None else cos.float().contiguous()
        sinf = None if sin is None else sin.float().contiguous()
        return tuple(N.ops().qknorm_rope_joint(tens, cosf, sinf, num_heads, eps))
    outs, off = [], 0
    for qkv, qs, ks in streams:
        L = qkv.shape[1]
        c = None if cos is None else cos[off:off + L]
        s_ = None if sin is None else sin[off:off + L]
        outs.append(R.qknorm_rope(qkv, qs, ks, c, s_, num_heads, eps))
        off += L
    if len(outs) == 1:
        return outs[0]
    return tuple(torch.cat([o[j] for o in outs], dim=1) for j in range(3))


# ---------------------------------------------------------------------------- gate + residual
def gate_residual(x, y, gate=None):
    if _native_ok(x, y, gate) and y.dim() == 3 and y.shape[-1] % 8 == 0:
        return N.ops().gate_residual(x, y, gate)
    return R.gate_residual(x, y, gate)


def split_tokens(x, n):
    """``(x[:, :n], x[:, n:])`` whose backward is a single concatenation."""
    if x.requires_grad and torch.is_grad_enabled() and x.is_cuda and _BACKEND == "fused":
        return tuple(N.ops().split_tokens(x, n))
    return x[:, :n], x[:, n:]


# ---------------------------------------------------------------------------- activations
def gelu_tanh(x):
    if _native_ok(x) and x.numel() % 8 == 0:
        return N.ops().act(x, 0)
    return R.gelu_tanh(x)


def silu(x):
    if _native_ok(x) and x.numel() % 8 == 0:
        return N.ops().act(x, 1)
    return R.silu(x)


def glu(h, mode="gelu", act_first=True):
    if _native_ok(h) and h.shape[-1] % 16 == 0:
        return N.ops().glu(h, 0 if mode == "gelu" else 1, act_first)
    return R.glu(h, mode, act_first)


# ---------------------------------------------------------------------------- GEMM family
_ACT_CODE = {None: 0, "gelu": 1, "silu": 2, "gelu_bwd": 3, "silu_bwd": 4}


def gemm_native(a, b, *, out=None, alpha=1.0, bias=None, lora_h=None, lora_b=None, act=None,
                pre_out=None, pre_in=None, residual=None, gate=None, rows_per_batch=0,
                n_split=0, out2=None, force_bn=0, b_mn=False, gather=None, scatter=None, pdl=False,
                a_mn=False, glu=0, _prepare_only=False):
    """out[M,N] = epilogue(a[M,K] @ op(b) (+ lora_h[M,r] @ lora_b[N,r]^T)) on the tcgen05 kernel.

    ``b`` is [N, K] (``op`` = transpose) or, with ``b_mn=True``, [K, N] used as is. ``a``/``b``/
    ``out`` may be row-strided views (last dim contiguous). ``gather``: dict built by
    ``parallel.gather_gemm`` (copy jobs + slab counters, fuses an operand gather into the launch).
    ``scatter``: dict(world, rank, part_cols, group_cols, local_rows, ptrs) routing column groups
    to peer buffers (``out`` is then only used for its row stride); with ``mode=1`` output ROW r goes to
    rank ``r // local_rows`` into slot ``rank`` of that rank's receive buffer ``[world][local_rows, N]``. ``a_mn=True``: ``a`` is [K, M]
    used as is (with ``b_mn`` this is the weight-gradient product over token-major activations).
    ``glu`` 1-4: ``b`` is an up-projection [2*hidden, K] and the output is the gated product of its
    halves, [M, hidden] (1 a*gelu(g), 2 a*silu(g), 3 gelu(a)*g, 4 silu(a)*g); ``pre_out``
    [M, 2*hidden] keeps the halves for backward. Returns ``out``.
    """
    lib = N.require()
    K, M = a.shape if a_mn else a.shape[::-1]
    Nn = b.shape[1] if b_mn else b.shape[0]
    assert (b.shape[0] if b_mn else b.shape[1]) == K and a.stride(1) == 1 and b.stride(1) == 1
    if out is None:
        cols = Nn // 2 if glu else (Nn if not n_split else n_split)
        out = torch.empty(M, cols, dtype=torch.bfloat16, device=a.device)
    g = N.GemmArgs()
    g.a, g.b = a.data_ptr(), b.data_ptr()
    g.lda, g.ldb = a.stride(0), b.stride(0)
    g.M, g.N, g.K = M, Nn, K
    g.alpha = alpha
    g.out, g.ldc = out.data_ptr(), out.stride(0)
    g.bias = N.ptr(bias)
    if lora_h is not None:
        g.lora_h, g.lora_b = lora_h.data_ptr(), lora_b.data_ptr()
        g.ld_h, g.ld_lb = lora_h.stride(0), lora_b.stride(0)
        g.lora_r = lora_h.shape[1]
    g.act = _ACT_CODE[act]
    if pre_out is not None:
        g.pre_out, g.ld_pre = pre_out.data_ptr(), pre_out.stride(0)
    if pre_in is not None:
        g.pre_in, g.ld_pre = pre_in.data_ptr(), pre_in.stride(0)
    if residual is not None:
        g.residual, g.ldr = residual.data_ptr(), residual.stride(0)
    if gate is not None:
        g.gate, g.gate_stride = gate.data_ptr(), gate.stride(0)
    g.rows_per_batch = rows_per_batch
    g.n_split = n_split
    if out2 is not None:
        g.out2, g.ldc2 = out2.data_ptr(), out2.stride(0)
    g.force_bn = force_bn
    if N.DEBUG_BOUNDS:
        g.dbg_out_bytes = N.extent_bytes(out) if scatter is None else 0
        g.dbg_out2_bytes, g.dbg_pre_bytes = N.extent_bytes(out2), N.extent_bytes(pre_out)
        g.dbg_res_bytes = N.extent_bytes(residual)
    g.b_mn = 1 if b_mn else 0
    g.a_mn = 1 if a_mn else 0
    g.glu = int(glu)
    g.pdl = 1 if (pdl and lora_h is not None and gather is None) else 0
    if gather is not None:
        g.n_copy, g.n_jobs = gather["n_copy"], gather["n_jobs"]
        g.jobs, g.flags, g.flag_target = gather["jobs"], gather["flags"], gather["flag_target"]
        g.b_flag_rows, g.a_flag_cols = gather.get("b_flag_rows", 0), gather.get("a_flag_cols", 0)
        g.rot_n_rows, g.rot_k_cols = gather.get("rot_n_rows", 0), gather.get("rot_k_cols", 0)
        g.a_flag_rows = gather.get("a_flag_rows", 0)
        g.all_flag = int(gather.get("all_flag", 0))
        st = gather.get("stamps")                 # optional uint64[8] phase record (see gemm_args.h)
        g.stamps = st.data_ptr() if st is not None else None
        # Copy clusters join the tile loop when their slabs have landed. The round from which the tile
        # schedule counts them in is the number of tiles a compute cluster finishes meanwhile: a copy
        # CTA moves ~35 GB/s (measured, bulk-copy ring), a K step of a pair tile is ~0.33 us.
        # Off unless asked for (``join_round`` in the plan's arguments, or ERI_B200_GATHER_JOIN=1): with
        # eight ranks emulated on one GPU it shortened the compute phase by one round of 13 but not the
        # launch as a whole.
        if gather.get("join_round") is not None:
            g.join_round = int(gather["join_round"])
        elif _GATHER_JOIN and g.n_copy > 0 and gather.get("copy_bytes"):
            copy_us = gather["copy_bytes"] / g.n_copy / 35e3
            tile_us = ((K + 63) // 64) * 0.33 + 2.0
            g.join_round = max(1, int(math.ceil(copy_us / tile_us)))
        loc = gather.get("local") if _GATHER_LOCAL else None
        if loc is not None:
            g.b_local, g.ldb_local = loc["ptr"], loc["ld"]
            g.loc_mode, g.loc_lo, g.loc_hi = loc["mode"], loc["lo"], loc["hi"]
            g.n_jobs_nl, g.jobs_nl, g.flag_target_nl = loc["n_jobs"], loc["jobs"], loc["flag_target"]
    if scatter is not None:
        g.scatter_world, g.scatter_rank = scatter["world"], scatter["rank"]
        g.scatter_part_cols, g.scatter_group_cols = scatter["part_cols"], scatter["group_cols"]
        g.scatter_local_rows = scatter["local_rows"]
        g.scatter_mode = int(scatter.get("mode", 0))
        for i, ptr_ in enumerate(scatter["ptrs"]):
            g.scatter_out[i] = ptr_
        if scatter.get("rowsq") is not None:
            g.rowsq, g.rowsq_parts = scatter["rowsq"].data_ptr(), scatter["rowsq"].shape[0]
    route = (M, Nn, K, a_mn, glu, gather, scatter, force_bn)
    if _prepare_only:
        return g, out, route          # ``gemm_native_pair`` launches it, alone or grouped
    return _launch_gemm(lib, g, out, route)


def _launch_gemm(lib, g, out, route):
    M, Nn, K, a_mn, glu, gather, scatter, force_bn = route
    # Few 128 x 128 tiles: the K range over a cluster, two CTAs per SM (answers -30 for any other product).
    if gather is None and scatter is None and force_bn <= 0 and (not a_mn or (M >= 256 and Nn >= 256)):
        code = lib.eri_gemm_few_bf16(g, N.stream_ptr())
        if code != -30:
            N.check(code, "gemm_few_bf16")
            return out
    # Few pair tiles (the 512-token text stream against a 3072-wide weight: 24 tiles for 74 CTA pairs)
    # leave most SMs idle; the one-CTA kernel's 128-column tiles spread the same work over four times
    # as many CTAs (measured 22.5 against 30.7 us at 512 x 3072 x 3072, 61 against 78 us at K = 12288).
    few_tiles = (force_bn == 0 and not (a_mn or glu) and gather is None and scatter is None
                 and ((M + 255) // 256) * ((Nn + 255) // 256) <= _PAIR_MIN_TILES)
    if (_GEMM_PAIR or a_mn or glu) and (gather is None or _GATHER_PAIR) and (scatter is None or _SCATTER_PAIR) \
            and force_bn in (0, 256) and M >= 256 and Nn >= 256 and not few_tiles:
        # two-CTA 256x256 tiles; in gather mode with whole copy clusters in front (answers -30 when
        # the gather plan does not line up with pair tiles, and the one-CTA kernel takes over)
        code = lib.eri_gemm2_bf16(g, N.stream_ptr())
        if code != -30:
            N.check(code, "gemm2_bf16")
            return out
    if a_mn or glu:
        raise ValueError(f"gemm_native: a_mn / glu need the two-CTA kernel's shape range (M={M}, N={Nn}, K={K})")
    code = lib.eri_gemm_bf16(g, N.stream_ptr())
    N.check(code, "gemm_bf16")
    return out


_GEMM_GROUP = os.environ.get("ERI_B200_GEMM_GROUP", "1") == "1"
_ACT_EPILOGUE = os.environ.get("ERI_B200_ACT_EPILOGUE", "0") == "1"   # activation + stored pre-activation in the GEMM epilogue


def _act_outside_epilogue(M, Nn, K) -> bool:
    """Whether a training-time linear + activation writes its pre-activation from the GEMM and applies the
    activation in a pass of its own. With a short reduction (K <= 4096) the epilogue of a pair tile is on the
    critical path and storing both tensors from it costs a large GEMM more than the separate pass
    ([4096 x 12288 x 3072]: 282 against 225 + 39 us); with a long reduction the epilogue is hidden, and a small
    problem is bound by its launches, so both keep the fused form."""
    return not _ACT_EPILOGUE and K <= 4096 and M * Nn >= (1 << 25)


def gemm_native_pair(kw0: dict, kw1: dict):
    """Two independent products (keyword arguments of ``gemm_native`` each) in ONE launch of the two-CTA
    kernel when they qualify: same N, K, operand majors, LoRA rank and epilogue kind, plain modes. The
    second problem's tiles follow the first's in the persistent schedule, so a small second problem
    (the text stream of a dual-stream block) runs in the first one's last, partly empty round instead of
    as a launch that leaves most SMs idle. Otherwise the two are launched one after the other.
    Returns (out0, out1)."""
    lib = N.require()
    g0, out0, r0 = gemm_native(**kw0, _prepare_only=True)
    g1, out1, r1 = gemm_native(**kw1, _prepare_only=True)
    plain = all(not (r[3] or r[4]) and r[5] is None and r[6] is None and r[7] == 0 and r[0] >= 256 and r[1] >= 256
                for r in (r0, r1))
    if _GEMM_GROUP and _GEMM_PAIR and plain and hasattr(lib, "eri_gemm2_bf16_group2"):
        code = lib.eri_gemm2_bf16_group2(g0, g1, N.stream_ptr())
        if code != -30:
            N.check(code, "gemm2_bf16_group2")
            return out0, out1
    return _launch_gemm(lib, g0, out0, r0), _launch_gemm(lib, g1, out1, r1)


def skinny_gemm(a, b, alpha=1.0):
    """alpha * a[M, K] @ b[N, K]^T for N in {16, 32, 64} (LoRA rank): split-K tcgen05 kernel that
    keeps every SM busy on a bandwidth-bound problem; other shapes use the general GEMM."""
    M, K = a.shape
    Nn = b.shape[0]
    lib = N.require()
    if _RANK_STREAM and hasattr(lib, "eri_gemm_rank_stream") and a.stride(1) == 1 and b.stride(1) == 1:
        # streaming kernel: bound by reading a once, no operand staging
        out = torch.empty(M, Nn, dtype=torch.bfloat16, device=a.device)
        code = lib.eri_gemm_rank_stream(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), out.data_ptr(),
                                        Nn, M, Nn, K, float(alpha), N.stream_ptr())
        if code != -100:
            N.check(code, "gemm_rank_stream")
            return out
    if hasattr(lib, "eri_gemm_skinny") and a.stride(1) == 1 and b.stride(1) == 1 and M >= 128:
        out = torch.empty(M, Nn, dtype=torch.bfloat16, device=a.device)
        code = lib.eri_gemm_skinny(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), out.data_ptr(),
                                   Nn, M, Nn, K, float(alpha), N.stream_ptr())
        if code != -100:
            N.check(code, "gemm_skinny")
            return out
    return gemm_native(a, b, alpha=alpha)


def skinny_gemm_pair(a0, b0, alpha0, a1, b1, alpha1):
    """(alpha0 * a0 b0^T, alpha1 * a1 b1^T) for two rank-r products with the same K and r (the adapters of the
    image and the text projection of a dual-stream block) in one launch of the streaming kernel; two
    launches when the shapes do not allow it."""
    lib = N.require()
    if (_RANK_STREAM and _GEMM_GROUP and hasattr(lib, "eri_gemm_rank_stream2") and a0.shape[1] == a1.shape[1]
            and b0.shape[0] == b1.shape[0] and all(t.stride(1) == 1 for t in (a0, b0, a1, b1))):
        r, K = b0.shape[0], a0.shape[1]
        o0 = torch.empty(a0.shape[0], r, dtype=torch.bfloat16, device=a0.device)
        o1 = torch.empty(a1.shape[0], r, dtype=torch.bfloat16, device=a1.device)
        code = lib.eri_gemm_rank_stream2(a0.data_ptr(), a0.stride(0), b0.data_ptr(), b0.stride(0), o0.data_ptr(), r,
                                         a0.shape[0], float(alpha0), a1.data_ptr(), a1.stride(0), b1.data_ptr(),
                                         b1.stride(0), o1.data_ptr(), r, a1.shape[0], float(alpha1), r, K,
                                         N.stream_ptr())
        if code != -100:
            N.check(code, "gemm_rank_stream2")
            return o0, o1
    return skinny_gemm(a0, b0, alpha=alpha0), skinny_gemm(a1, b1, alpha=alpha1)


def gemm_supported(M, Nn, K) -> bool:
    return M >= 128 and Nn >= 16 and K >= 8 and K % 8 == 0 and Nn % 8 == 0


def set_gemm_pair(on: bool) -> None:
    global _GEMM_PAIR
    _GEMM_PAIR = bool(on)


def gemm_error_check() -> int:
    """Synchronise and return the device error word of the GEMM kernels (0 = clean)."""
    return next(iter(N.error_words(("gemm", "gemm2", "gemm_few")).values()), 0)


def kernel_error_check() -> dict:
    """Synchronise and read every kernel family's device error word (each is set when one of that
    family's bounded waits ran out, and cleared by the read). Empty dict = clean."""
    return N.error_words()


def _wgrad_ok(*ts) -> bool:
    return _WGRAD_NATIVE and _BACKEND == "fused" and _GEMM_NATIVE == "native" and all(
        t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1
        and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in ts)


def wgrad(dy2, x2, accum=None, out=None):
    """Weight gradient dW[N_out, K_in] = dy2[T, N_out]^T @ x2[T, K_in] on the two-CTA tcgen05 kernel:
    both activations are read token-major as MN-major operands, so no transposed copy is made.
    ``accum``: an existing bf16 gradient of that shape; the product is added into it (beta = 1 in the
    GEMM epilogue) and ``accum`` is returned. ``out``: destination for the plain product. Shapes
    outside the kernel's range use ``torch``."""
    T, Nn = dy2.shape
    K = x2.shape[1]
    dst = accum if accum is not None else out
    if _wgrad_ok(dy2, x2) and Nn >= 256 and K >= 256 and T >= 64 and Nn % 8 == 0 and K % 8 == 0 \
            and (dst is None or _wgrad_ok(dst)):
        return gemm_native(dy2, x2, a_mn=True, b_mn=True, out=dst, residual=accum)
    if accum is not None:
        return accum.addmm_(dy2.t(), x2)
    if out is not None:
        return torch.mm(dy2.t(), x2, out=out)
    return dy2.t() @ x2


def lora_wgrad(a_tok, b_tok, out=None, transpose_out=False, accumulate=False):
    """Skinny token reduction ``a_tok[T, Mg]^T @ b_tok[T, r]`` (r = adapter rank) for the LoRA
    gradients: dB[N_out, r] = dY^T H, and with ``transpose_out`` dA[r, K_in] = (X^T Ts)^T. Split over
    the tokens across CTAs on tcgen05; ``accumulate`` adds into ``out``."""
    T, Mg = a_tok.shape
    r = b_tok.shape[1]
    shape = (r, Mg) if transpose_out else (Mg, r)
    lib = N.lib() if a_tok.is_cuda else None
    if lib is not None and hasattr(lib, "eri_gemm_tokred") and _wgrad_ok(a_tok) and r in (16, 32, 64) \
            and b_tok.is_cuda and b_tok.dtype == torch.bfloat16 and b_tok.stride(1) == 1 and b_tok.stride(0) % 8 == 0 \
            and b_tok.data_ptr() % 16 == 0 and T >= 64 and Mg >= 128 and Mg % 8 == 0 \
            and (out is None or (out.dtype == torch.bfloat16 and out.stride(1) == 1 and tuple(out.shape) == shape)):
        if out is None:
            out, accumulate = torch.empty(shape, dtype=torch.bfloat16, device=a_tok.device), False
        code = lib.eri_gemm_tokred(a_tok.data_ptr(), a_tok.stride(0), b_tok.data_ptr(), b_tok.stride(0),
                                   out.data_ptr(), out.stride(0), T, Mg, r, 1.0, 1 if transpose_out else 0,
                                   1 if accumulate else 0, N.extent_bytes(out) if N.DEBUG_BOUNDS else 0,
                                   N.stream_ptr())
        if code != -100:
            N.check(code, "gemm_tokred")
            return out
    prod = b_tok.t() @ a_tok if transpose_out else a_tok.t() @ b_tok
    if out is None:
        return prod
    return out.add_(prod) if accumulate else out.copy_(prod)


_ACCUM_INTO_GRAD = os.environ.get("ERI_B200_ACCUM_INTO_GRAD", "1") == "1"


def _flags(x=None, w=None, act=None) -> int:
    """The switches of this module that the native nodes honour (``Flag`` in csrc/torch/eri_ops.h), with the rule for the
    activation of a linear ``act(x w^T)``."""
    outside = act is not None and x.shape[-1] > 0 and _act_outside_epilogue(x.numel() // x.shape[-1], w.shape[0], x.shape[-1])
    return ((1 if _pdl_ok() else 0) | (2 if _RANK_STREAM else 0) | (4 if _GEMM_PAIR else 0) | (8 if _GEMM_GROUP else 0)
            | (16 if outside else 0) | (32 if _WGRAD_NATIVE else 0) | (64 if _ACCUM_INTO_GRAD else 0)
            | (128 if _GEMM_NATIVE == "native" else 0) | (max(0, min(_PAIR_MIN_TILES, 1 << 20)) << 8))


def prepare_lora_transposes(matrices):
    """Transpose every adapter matrix of a model in ONE launch and publish the copies for this
    step's backward (which needs B^T for ``dY B`` and A^T as the rank-r K-step operand). Without
    this each adapted linear transposes its two small matrices itself: two extra launches per
    site per step. Call once per step after the optimizer update, before backward."""
    if _BACKEND != "fused" or not any(m.is_cuda for m in matrices):
        return 0
    return N.ops().prepare_lora_transposes(list(matrices))


def invalidate_lora_transposes(matrices=()):
    """The adapter matrices changed (optimizer step): the published transposes of every set that one of ``matrices``
    belongs to (default: of every set) are stale."""
    if N._ops is not None:
        N._ops.invalidate_lora_transposes(list(matrices))


def _lora_transposed(m):
    return N.ops().lora_transposed(m)


def linear(x, w, bias=None, lora=None, act=None, residual=None, gate=None, wt=None):
    """Fused linear. lora = (A [r,K], B [N,r], scale) or None; act in {None,"gelu","silu"};
    residual [.., N] and gate [B, N] give ``residual + gate * y``. Saved for backward: x, the rank-r
    product, the pre-activation (when act); never a materialised LoRA delta. ``wt`` is an optional
    cached transpose of a frozen W ([K, N]) that lets the input-gradient GEMM read a K-major operand."""
    if _BACKEND == "fused" and x.is_cuda:
        a, b, s = lora if lora is not None else (None, None, 1.0)
        y = N.ops().linear(x, w, bias, a, b, s, _ACT_CODE[act], residual, gate, wt, _flags(x, w, act))
        if y is not None:
            return y
    y = R.linear(x, w, bias, lora, act, None, None)
    if gate is not None or residual is not None:
        y = R.gate_residual(residual, y, gate)
    return y


def _linear_pair_ok(x0, lin0, x1, lin1) -> bool:
    (w0, b0, lo0, r0, g0), (w1, b1, lo1, r1, g1) = lin0, lin1

    def rank_ok(lo):
        return lo is None or lo[0].shape[0] in (16, 32, 64)
    return bool(_GEMM_GROUP and _GEMM_NATIVE == "native" and _native_ok(x0, w0, b0) and _native_ok(x1, w1, b1)
                and w0.shape == w1.shape and x0.shape[-1] % 8 == 0 and rank_ok(lo0) and rank_ok(lo1)
                and (lo0 is None) == (lo1 is None) and (lo0 is None or lo0[0].shape[0] == lo1[0].shape[0])
                and (b0 is None) == (b1 is None)
                and x0.numel() // x0.shape[-1] >= 256 and x1.numel() // x1.shape[-1] >= 256
                and gemm_supported(x0.numel() // x0.shape[-1], w0.shape[0], x0.shape[-1])
                and gemm_supported(x1.numel() // x1.shape[-1], w1.shape[0], x1.shape[-1]))


def linear_pair_ok(x0, lin0, x1, lin1) -> bool:
    """Whether ``linear_pair`` would run the two layers as grouped launches."""
    return _linear_pair_ok(x0, lin0, x1, lin1)


def linear_pair(x0, lin0, x1, lin1, act=None, emit_pre=False, act_in=None, x_pre=(None, None)):
    """``lin_i`` = (w, bias, lora or None, residual or None, gate or None). Returns (y0, y1) of two fused
    linears whose main GEMMs (and input-gradient GEMMs) share one launch when both run on the native path
    with matching shapes; otherwise exactly ``linear`` twice. ``emit_pre`` / ``act_in`` + ``x_pre`` (only
    when ``linear_pair_ok``): see ``FusedLinearPair`` in csrc/torch/gemm_ops.cpp; with ``emit_pre`` the result is
    (pre_0, pre_1, act(pre_0), act(pre_1))."""
    (w0, b0, lo0, r0, g0), (w1, b1, lo1, r1, g1) = lin0, lin1
    def apply(rg0, rg1):
        a0, bb0, s0 = lo0 if lo0 is not None else (None, None, 1.0)
        a1, bb1, s1 = lo1 if lo1 is not None else (None, None, 1.0)
        return tuple(N.ops().linear_pair([x0, x_pre[0], w0, b0, a0, bb0, *rg0], s0, [x1, x_pre[1], w1, b1, a1, bb1, *rg1],
                                         s1, _ACT_CODE[act], emit_pre, _ACT_CODE[act_in],
                                         _flags(x0, w0, act)))

    if emit_pre or act_in is not None:
        return apply((r0, g0), (r1, g1))
    if not _linear_pair_ok(x0, lin0, x1, lin1):
        return (linear(x0, w0, b0, lora=lo0, act=act, residual=r0, gate=g0),
                linear(x1, w1, b1, lora=lo1, act=act, residual=r1, gate=g1))
    if (g0 is not None and g0.requires_grad) or (g1 is not None and g1.requires_grad):
        # trainable modulation: the gates stay outside the GEMM epilogue so that their gradients are produced
        y0, y1 = apply((None, None), (None, None))
        return gate_residual(r0, y0, g0), gate_residual(r1, y1, g1)
    return apply((r0, g0), (r1, g1))


_GLU_FUSED = os.environ.get("ERI_B200_GLU_FUSED", "1") == "1"
_GLU_CODE = {("gelu", False): 1, ("silu", False): 2, ("gelu", True): 3, ("silu", True): 4}


def linear_glu(x, lin, mode="gelu", act_first=True):
    """``glu(lin(x), mode, act_first)`` for an up-projection module ``lin`` ([2*hidden, K] weight).
    One GEMM launch with the gate in its epilogue when the shape fits the two-CTA kernel and the
    adapter (if any) is a plain LoRA; otherwise the projection and the gate run as separate ops."""
    ad = getattr(lin, "adapter", None)
    w, b = lin.weight, lin.bias
    rows = x.numel() // x.shape[-1]
    plain_lora = ad is not None and getattr(ad, "kind", "") == "lora" and ad.rank in (16, 32, 64) \
        and not (ad.dropout > 0 and ad.training)
    if _GLU_FUSED and _GEMM_NATIVE == "native" and _native_ok(x, w, b) and (ad is None or plain_lora) \
            and type(lin).__name__ == "Linear" and rows >= 256 and w.shape[0] >= 256 and w.shape[0] % 16 == 0 \
            and x.shape[-1] % 8 == 0 and x.shape[-1] >= 64:
        wt = lin.frozen_transpose() if torch.is_grad_enabled() else None
        a, bb, s = (ad.lora_A, ad.lora_B, float(ad.scale)) if ad is not None else (None, None, 1.0)
        return N.ops().linear_glu(x, w, b, a, bb, s, _GLU_CODE[(mode, bool(act_first))], wt, _flags())
    return glu(lin(x), mode, act_first)


def _rows_ok(*ts):
    return all(t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0
               and t.data_ptr() % 16 == 0 for t in ts)


def small_wgrad(dy2, xin, scale: float = 1.0):
    """dW[N, K] = scale * dy2[T, N]^T @ xin[T, K] for a handful of rows (T <= 8): one pass that is
    bound by writing dW (native kernel); other shapes use ``torch``."""
    T, Nn = dy2.shape
    K = xin.shape[1]
    lib = N.lib() if dy2.is_cuda else None
    if lib is not None and _BACKEND == "fused" and hasattr(lib, "eri_rows_wgrad") and T <= 8 and K % 8 == 0 \
            and _rows_ok(xin) and dy2.dtype == torch.bfloat16 and dy2.stride(1) == 1:
        return N.ops().small_wgrad(dy2, xin, float(scale))
    dw = dy2.t() @ xin
    return dw if scale == 1.0 else dw * scale


def small_dgrad(dy2, w):
    """dx[T, K] = dy2[T, N] @ w[N, K] for T <= 8: one pass over w split across CTAs by rows of w; the
    fp32 partial planes are added in split order (deterministic)."""
    T, Nn = dy2.shape
    K = w.shape[1]
    lib = N.lib() if dy2.is_cuda else None
    if lib is not None and _BACKEND == "fused" and hasattr(lib, "eri_rows_dgrad") and T <= 8 and K % 8 == 0 \
            and _rows_ok(w) and dy2.dtype == torch.bfloat16 and dy2.stride(1) == 1:
        return N.ops().small_dgrad(dy2, w)
    return dy2 @ w


def small_linear(x, w, bias=None, silu_in=False):
    """Linear on a handful of rows (adaLN modulation and embedders); SiLU on the input optional."""
    rows = x.numel() // x.shape[-1]
    if _native_ok(x, w, bias) and rows <= 8 and x.shape[-1] % 8 == 0 and x.shape[-1] * rows <= 50000:
        return N.ops().small_linear(x, w, bias, silu_in, _ACCUM_INTO_GRAD)
    xin = torch.nn.functional.silu(x) if silu_in else x
    return torch.nn.functional.linear(xin, w, bias)


# ---------------------------------------------------------------------------- attention
# read once at import: the ATTN_* switches of the library attention path (utils/env_flags.py)
_ATTN_ENV_POLICY = any(os.environ.get(k) for k in ("ATTN_Q_CHUNK", "ATTN_KV_CHUNK", "ATTN_MAX_WS_MB", "ATTN_MIN_FREE_MB"))


_HEAD_PAD = os.environ.get("ERI_B200_ATTN_HEAD_PAD", "1") == "1"
ATTENTION_CALLS = {"native": 0, "library": 0}     # forward calls by path since import (benchmarks print it)


def attention(q, k, v, scale=None, mask=None, out=None):
    """Non-causal attention over token-major [B, L, H, Dh] tensors. ``out``: optional destination
    buffer for the native kernel (ignored by the library path, which returns its own tensor)."""
    if _ATTN_NATIVE == "native" and _native_ok(q, k, v):
        from . import flash_attn as FA
        # key-only masks (text padding, [B, 1, 1, T]) ride on the native kernel as a per-key bias
        if FA.supported(q, k, v, strided=out is None) and (mask is None or FA.mask_is_key_only(mask, q.shape[0], k.shape[1])):
            ATTENTION_CALLS["native"] += 1
            return FA.flash_attention(q, k, v, scale, out, mask)
        if mask is None and out is None and _wide_ok(q, k, v, scale):
            ATTENTION_CALLS["native"] += 1
            return N.ops().attention_wide(q, k, v, scale if scale is not None else 1.0 / math.sqrt(512))
        if mask is not None and out is None and _bias_ok(q, k, v, mask):
            ATTENTION_CALLS["native"] += 1
            return N.ops().attention_bias(q, k, v, mask, scale if scale is not None else 1.0 / math.sqrt(q.shape[-1]))
        # other head sizes below 128 (SD1.5: 40 and 80) ride on the 64 / 128 kernels with zero columns
        # appended: zero query / key columns leave the scores unchanged, zero value columns give zero
        # output columns that are cut off again (the pad and the slice are differentiable copies)
        D = q.shape[-1]
        if _HEAD_PAD and D not in (64, 128) and 16 <= D < 128 and D % 8 == 0 and \
                (mask is None or FA.mask_is_key_only(mask, q.shape[0], k.shape[1])):
            pad = (64 if D < 64 else 128) - D
            qp, kp, vp = (torch.nn.functional.pad(t, (0, pad)) for t in (q, k, v))
            if FA.supported(qp, kp, vp):
                ATTENTION_CALLS["native"] += 1
                sc = scale if scale is not None else 1.0 / math.sqrt(D)
                return FA.flash_attention(qp, kp, vp, sc, None, mask)[..., :D].contiguous()
    ATTENTION_CALLS["library"] += 1
    if mask is None and _ATTN_ENV_POLICY:
        from ..utils.env_flags import library_attention
        o = library_attention(q, k, v, scale)
        if o is not None:
            return o
    return R.attention(q, k, v, scale, mask)


_GRID_YZ = 65535       # blocks in the second and third dimension of a launch


def _wide_ok(q, k, v, scale) -> bool:
    """Head size 512 (the image autoencoders' middle block), forward only: tiles of 128 queries and 128 keys. The kernel
    takes a row's maximum before it scales, so a negative scale is the library's."""
    return (q.shape[-1] == 512 and (scale is None or scale >= 0) and 1 <= q.shape[0] <= _GRID_YZ and 1 <= q.shape[2] <= _GRID_YZ
            and q.shape[1] >= 128 and k.shape[1] >= 128 and k.shape == v.shape and q.shape[0] == k.shape[0]
            and q.shape[2] == k.shape[2] and not (torch.is_grad_enabled() and any(t.requires_grad for t in (q, k, v))))


def _bias_ok(q, k, v, mask) -> bool:
    """A mask per query and key (relative-position bias, causal), forward only: bf16 or boolean, a value for every key."""
    B, Lq, H, D = q.shape
    return (D in (64, 128) and 1 <= B <= _GRID_YZ and 1 <= H <= _GRID_YZ and Lq >= 1 and k.shape[1] >= 1
            and k.shape == v.shape == (B, k.shape[1], H, D) and mask.device == q.device
            and mask.dtype in (torch.bool, torch.bfloat16) and mask.dim() == 4 and mask.shape[3] == k.shape[1]
            and mask.shape[0] in (1, B) and mask.shape[1] in (1, H) and mask.shape[2] in (1, Lq)
            and not (torch.is_grad_enabled() and any(t.requires_grad for t in (q, k, v, mask))))


def _packed_ok(head_dim, mask, B, Lk, *ts) -> bool:
    from . import flash_attn as FA
    return (_ATTN_NATIVE == "native" and head_dim in (64, 128) and _native_ok(*ts) and ts[0].shape[1] >= 16 and Lk >= 1 and FA.has_forward()
            and (mask is None or FA.mask_is_key_only(mask, B, Lk)))


def attention_qkv(qkv, num_heads, scale=None, mask=None):
    """Self-attention on a packed projection [B, L, 3*H*Dh] -> [B, L, H*Dh]. On the native path q, k and v are read
    in place and the gradient is written as one packed tensor."""
    B, L, W = qkv.shape
    Dh = W // (3 * num_heads)
    if _packed_ok(Dh, mask, B, L, qkv):
        from . import flash_attn as FA
        ATTENTION_CALLS["native"] += 1
        kb = None if mask is None else FA.key_bias(mask, B, L, qkv.device)
        return N.ops().attention_qkv(qkv, num_heads, scale if scale is not None else 1.0 / math.sqrt(Dh), kb)
    q, k, v = qkv.view(B, L, 3, num_heads, Dh).unbind(2)
    return attention(q.contiguous(), k.contiguous(), v.contiguous(), scale, mask).reshape(B, L, W // 3)


def attention_kv(q, kv, num_heads, scale=None, mask=None):
    """Cross-attention of q [B, L, H*Dh] on a packed key / value projection [B, Lk, 2*H*Dh] -> [B, L, H*Dh]."""
    B, L, W = q.shape
    Lk, Dh = kv.shape[1], W // num_heads
    if kv.shape[0] == B and kv.shape[2] == 2 * W and _packed_ok(Dh, mask, B, Lk, q, kv):
        from . import flash_attn as FA
        ATTENTION_CALLS["native"] += 1
        kb = None if mask is None else FA.key_bias(mask, B, Lk, q.device)
        return N.ops().attention_kv(q, kv, num_heads, scale if scale is not None else 1.0 / math.sqrt(Dh), kb)
    k, v = kv.view(B, Lk, 2, num_heads, Dh).unbind(2)
    return attention(q.view(B, L, num_heads, Dh), k.contiguous(), v.contiguous(), scale, mask).reshape(B, L, W)


def attention_qkv_rope(qkv, q_weight, k_weight, cos, sin, num_heads, eps=1e-6):
    """Self-attention on a packed projection [B, L, 3*H*Dh] whose queries and keys are first normalised (RMS over all
    H*Dh channels, times ``q_weight`` / ``k_weight``) and rotated over interleaved pairs of the whole width (cos / sin
    [L, H*Dh/2]) -> [B, L, H*Dh]. One kernel reads q, k and the tables once; trainable norm weights use the separate ops."""
    B, L, W = qkv.shape
    D = W // 3
    if _packed_ok(D // num_heads, None, B, L, qkv, q_weight, k_weight) and D % 8 == 0 and D <= 8192 and cos.is_cuda and sin.is_cuda \
            and cos.shape == sin.shape == (L, D // 2) \
            and not (torch.is_grad_enabled() and any(t.requires_grad for t in (q_weight, k_weight, cos, sin))):
        ATTENTION_CALLS["native"] += 1
        return N.ops().attention_qkv_rope(qkv, q_weight, k_weight, cos, sin, num_heads, eps)
    q, k, v = qkv.split(D, dim=-1)
    sh = (B, L, num_heads, D // num_heads)
    q, k = (R.rope_rotate(norm_modulate(t.contiguous(), weight=w, rms=True, eps=eps).unsqueeze(2), cos, sin).squeeze(2).to(t.dtype)
            for t, w in ((q, q_weight), (k, k_weight)))
    return attention(q.view(sh), k.view(sh), v.contiguous().view(sh)).reshape(B, L, D)


# ---------------------------------------------------------------------------- losses / noise
def mse_loss(pred, target, weight=None):
    """mean(weight[b] * (pred - target)^2) with the gradient produced in the same pass."""
    if _native_ok(pred, target) and pred.numel() % 8 == 0 and (pred.numel() // pred.shape[0]) % 8 == 0:
        return N.ops().mse_loss(pred, target, weight)
    return R.mse(pred, target, weight)


def noise_mix(x0, coef, seed: int, offset: int = 0, eps=None, patch=2, want_eps=False):
    """Build x_t and the regression target from clean latents in one pass.

    x0 [B, C, H, W]; coef [4, B] fp32 rows (a, s, ca, cb): x_t = a*x0 + s*eps,
    target = ca*eps + cb*x0. Noise comes from a Philox counter stream (seed, offset) unless
    ``eps`` is given. Returns token-major (x_t, target[, eps]) of shape [B, HW/p^2, C*p*p].
    """
    B, C, H, W = x0.shape
    if _native_ok(x0, eps) and (B * C * H * W) % 4 == 0:
        x0 = _c(x0)
        L, D = (H // patch) * (W // patch), C * patch * patch
        xt = torch.empty(B, L, D, dtype=x0.dtype, device=x0.device)
        tg = torch.empty_like(xt)
        eo = torch.empty_like(xt) if want_eps else None
        cf = coef.float().contiguous()
        N.check(N.require().eri_noise_mix(x0.data_ptr(), N.ptr(_c(eps)), cf.data_ptr(),
                                          xt.data_ptr(), tg.data_ptr(), N.ptr(eo), B, C, H, W,
                                          patch, seed, offset, N.stream_ptr()), "noise_mix")
        return (xt, tg, eo) if want_eps else (xt, tg)
    if eps is None:
        gen = torch.Generator(device=x0.device).manual_seed(seed + offset)
        eps = torch.randn(x0.shape, generator=gen, device=x0.device, dtype=torch.float32).to(x0.dtype)
    xt, tg = R.noise_mix(x0, eps, coef, patch)
    return (xt, tg, R.patchify(eps, patch)) if want_eps else (xt, tg)


def randn_bf16(shape, seed: int, offset: int = 0, device="cuda", mean=0.0, std=1.0):
    out = torch.empty(shape, dtype=torch.bfloat16, device=device)
    if out.is_cuda and _BACKEND == "fused":
        N.check(N.require().eri_randn_bf16(out.data_ptr(), out.numel(), seed, offset, mean, std,
                                           N.stream_ptr()), "randn")
        return out
    gen = torch.Generator(device=out.device).manual_seed(seed + offset)
    return (torch.randn(shape, generator=gen, device=out.device) * std + mean).to(torch.bfloat16)


def sumsq(flat, out=None):
    """Sum of squares of a flat bf16 buffer into a device fp32 scalar (no host sync)."""
    if out is None:
        out = torch.zeros((), dtype=torch.float32, device=flat.device)
    else:
        out.zero_()
    if _native_ok(flat):
        N.check(N.require().eri_sumsq_bf16(flat.data_ptr(), flat.numel(), out.data_ptr(),
                                           N.stream_ptr()), "sumsq")
    else:
        out.add_(flat.float().pow(2).sum())
    return out


# ---------------------------------------------------------------------------- GroupNorm (+SiLU)
def group_norm_silu(x, weight, bias=None, groups=32, eps=1e-5, silu=True, pre_c=None, pre_nc=None):
    """GroupNorm followed by an optional SiLU on a channels-last activation. ``x`` is either
    [N, HW, C] or an [N, C, H, W] tensor in ``torch.channels_last`` memory format (returned in the
    same logical shape and format). ``pre_c`` [C] and ``pre_nc`` [N, C] are added to x before the norm (the
    bias of the convolution that produced x and a per-sample embedding), in the same pass on the native path."""
    C = x.shape[1] if x.dim() == 4 else x.shape[-1]
    if _native_ok(x, weight, bias, pre_c, pre_nc) and C % 8 == 0 and C % groups == 0 and C <= 8192 and groups <= 4096:
        return N.ops().group_norm_silu(x, weight, bias, pre_c, pre_nc, groups, eps, silu, _ACCUM_INTO_GRAD)
    nchw = x.dim() == 4
    if nchw:
        Nn, C, H, W = x.shape
        rows = x.permute(0, 2, 3, 1)
        if not rows.is_contiguous():
            rows = rows.contiguous()
        rows = rows.view(Nn, H * W, C)
    else:
        rows = x
    if pre_c is not None:
        rows = rows + pre_c
    if pre_nc is not None:
        rows = rows + pre_nc[:, None, :]
    y = R.group_norm_silu(rows, weight, bias, groups, eps, silu)
    if nchw:
        return y.view(Nn, H, W, C).permute(0, 3, 1, 2)
    return y


def add_bias(a, b, bias=None, bias2=None):
    """``a + b`` plus per-channel biases: the residual sum of a convolutional block with the biases of its last
    convolutions. [N, HW, C] or channels-last [N, C, H, W]."""
    C = a.shape[1] if a.dim() == 4 else a.shape[-1]
    if _native_ok(a, b, bias, bias2) and C % 8 == 0 and a.shape == b.shape:
        return N.ops().add_bias(a, b, bias, bias2, _ACCUM_INTO_GRAD)
    y = a + b
    for t in (bias, bias2):
        if t is not None:
            y = y + (t[:, None, None] if a.dim() == 4 else t)
    return y


def upsample2x(x):
    """Nearest-neighbour upsampling by two of an [N, C, H, W] activation (channels-last on the native path)."""
    if _native_ok(x) and x.dim() == 4 and x.shape[1] % 8 == 0:
        return N.ops().upsample2x(x)
    return torch.nn.functional.interpolate(x, scale_factor=2.0, mode="nearest")


def unhooked(*modules) -> bool:
    """Whether nobody listens to these modules' calls (forward or backward hooks, a replaced ``forward``): only then may
    their work be done without calling them, or be handed other arguments than they would see."""
    return all(not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                    or "forward" in m.__dict__) for m in modules)


def conv_fusable(x, *convs) -> bool:
    """Whether the biases of ``convs`` may be added by the ops around them (``group_norm_silu``'s ``pre_c``,
    ``add_bias``) instead of in a pass after each convolution: plain convolutions on the native path."""
    return _native_ok(x) and all(c is None or (type(c) is torch.nn.Conv2d and unhooked(c) and c.padding_mode == "zeros"
                                               and c.out_channels % 8 == 0) for c in convs)


def conv_no_bias(conv, x):
    """``conv(x)`` without its bias. A 1x1 convolution runs as a linear on the pixel rows."""
    w = conv.weight
    if conv.kernel_size == (1, 1) and conv.stride == (1, 1) and conv.padding == (0, 0) and conv.groups == 1 \
            and x.shape[1] % 8 == 0:
        Nn, C, H, W = x.shape
        rows = x.permute(0, 2, 3, 1).reshape(Nn, H * W, C)
        return linear(rows, w.view(w.shape[0], C)).view(Nn, H, W, w.shape[0]).permute(0, 3, 1, 2)
    if torch.is_grad_enabled() and w.requires_grad and _native_ok(x, w) and conv.groups == 1 and not isinstance(conv.padding, str) \
            and w.is_contiguous() and w.shape[1] % 8 == 0 and w.shape[0] <= 65535 and 1 < w.shape[2] * w.shape[3] <= 25 \
            and w.data_ptr() % 16 == 0:
        # (a parameter of the flat arena; a weight already in channels-last order needs no copy)
        return N.ops().conv2d_trained(x, w, list(conv.stride), list(conv.padding), list(conv.dilation), _ACCUM_INTO_GRAD)
    return torch.nn.functional.conv2d(x, w, None, conv.stride, conv.padding, conv.dilation, conv.groups)


# ---------------------------------------------------------------------------- token routing
def token_scores(x):
    """L2 norm of every token row of x [B, L, D] -> fp32 [B, L]."""
    if _native_ok(x) and x.shape[-1] % 8 == 0:
        x = _c(x)
        out = torch.empty(x.shape[:-1], dtype=torch.float32, device=x.device)
        N.check(N.require().eri_row_l2norm(x.data_ptr(), out.data_ptr(), out.numel(), x.shape[-1],
                                           N.stream_ptr()), "row_l2norm")
        return out
    return x.float().norm(dim=-1)


def topk_indices(scores, k):
    """Indices [B, k] (int64) of the k largest non-negative scores per row, descending, ties by
    lower index; selection runs on the device (no host sort)."""
    B, L = scores.shape
    if scores.is_cuda and _BACKEND == "fused" and L <= 16384 and scores.dtype == torch.float32:
        idx = torch.empty(B, k, dtype=torch.int32, device=scores.device)
        N.check(N.require().eri_topk_desc(_c(scores).data_ptr(), idx.data_ptr(), B, L, k, N.stream_ptr()), "topk")
        return idx.long()
    return scores.topk(k, dim=1).indices


class _GatherRows(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, idx32):
        B, L, D = x.shape
        k = idx32.shape[1]
        x = _c(x)
        out = torch.empty(B, k, D, dtype=x.dtype, device=x.device)
        N.check(N.require().eri_gather_rows(x.data_ptr(), idx32.data_ptr(), out.data_ptr(), B, L, k, D,
                                            N.stream_ptr()), "gather_rows")
        ctx.save_for_backward(idx32)
        ctx.L = L
        return out

    @staticmethod
    def backward(ctx, dy):
        (idx32,) = ctx.saved_tensors
        B, k, D = dy.shape
        L = ctx.L
        dy = _c(dy)
        lib = N.require()
        inv = torch.full((B, L), -1, dtype=torch.int32, device=dy.device)
        N.check(lib.eri_build_inverse(idx32.data_ptr(), inv.data_ptr(), B, L, k, N.stream_ptr()), "build_inverse")
        dx = torch.empty(B, L, D, dtype=dy.dtype, device=dy.device)
        N.check(lib.eri_reinject_rows(None, dy.data_ptr(), inv.data_ptr(), dx.data_ptr(), B, L, k, D,
                                      N.stream_ptr()), "scatter_rows")
        return dx, None


class _ReinjectRows(torch.autograd.Function):
    @staticmethod
    def forward(ctx, full, routed, idx32):
        B, L, D = full.shape
        k = idx32.shape[1]
        full, routed = _c(full), _c(routed)
        lib = N.require()
        inv = torch.full((B, L), -1, dtype=torch.int32, device=full.device)
        N.check(lib.eri_build_inverse(idx32.data_ptr(), inv.data_ptr(), B, L, k, N.stream_ptr()), "build_inverse")
        out = torch.empty_like(full)
        N.check(lib.eri_reinject_rows(full.data_ptr(), routed.data_ptr(), inv.data_ptr(), out.data_ptr(),
                                      B, L, k, D, N.stream_ptr()), "reinject_rows")
        ctx.save_for_backward(idx32, inv)
        return out

    @staticmethod
    def backward(ctx, dy):
        idx32, inv = ctx.saved_tensors
        B, L, D = dy.shape
        k = idx32.shape[1]
        dy = _c(dy)
        lib = N.require()
        d_routed = torch.empty(B, k, D, dtype=dy.dtype, device=dy.device)
        N.check(lib.eri_gather_rows(dy.data_ptr(), idx32.data_ptr(), d_routed.data_ptr(), B, L, k, D,
                                    N.stream_ptr()), "gather_rows")
        d_full = dy * (inv < 0).unsqueeze(-1).to(dy.dtype)
        return d_full, d_routed, None


def gather_rows(x, idx):
    """x [B, L, D], idx [B, k] -> [B, k, D]."""
    if _native_ok(x) and x.shape[-1] % 8 == 0:
        return _GatherRows.apply(x, idx.to(torch.int32).contiguous())
    return torch.gather(x, 1, idx.long().unsqueeze(-1).expand(-1, -1, x.shape[-1]))


def reinject_rows(full, routed, idx):
    """Copy of ``full`` [B, L, D] whose rows ``idx`` [B, k] are replaced by ``routed`` [B, k, D]."""
    if _native_ok(full, routed) and full.shape[-1] % 8 == 0:
        return _ReinjectRows.apply(full, routed, idx.to(torch.int32).contiguous())
    return full.scatter(1, idx.long().unsqueeze(-1).expand(-1, -1, full.shape[-1]), routed)
