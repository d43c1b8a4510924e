// Flash attention forward with a mask of its own per query and key: softmax(scale * Q K^T + bias) V, head size 64 or
// 128, bf16 in / bf16 out. The bias is bf16 or boolean (false: -inf) with any broadcast over batch, head and query: the
// relative-position bias of T5-style encoders, the causal mask of CLIP-style ones. No gradient.
//
// The scores, the bias sum, the exponentials and the row sums are fp32, and a probability enters the second product
// as three bf16 terms (its rounding, the rounding of the rest, and what is left): all 24 bits of its mantissa, so the
// product is that of fp32 probabilities. One CTA per (128 queries, head, batch), two per SM at head size 64, as
// flash_attn.cu:
//   warp 0     TMA: Q once, then one K and one V tile of 128 keys per iteration
//   warp 1     tcgen05.mma issue: S = Q K^T, O += P1 V, O += P2 V, O += P3 V (P1 and P2 lie over S in TMEM, P3 has 64
//              columns of its own)
//   warps 2-9  softmax, two threads per query row, 64 keys of a tile each
// What bounds it: latency. At 256 tokens x 64 heads 128 CTAs run two tiles each, and a thread's bias row of 64 keys is
// one 128-byte line. The library ran this as fp32 products on the CUDA cores with separate bias, masking, softmax
// and conversion passes: about 110 us per layer.
#include "attn_args.h"
#include "ptx.cuh"
#include "tma_host.h"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

struct BiasParams {
  int B, H, Lq, Lk;
  float scale;
  bf16* out;              // [B, Lq, H, DH] contiguous
  const void* bias;       // element (b, h, q, k) at b * sb + h * sh + q * sq + k
  long long sb, sh, sq;
  int is_bool, vec;       // vec: bf16 rows readable in 16-byte words
  int* err;
};

constexpr int BQ = 128, BKV = 128;
constexpr float kRescaleThreshold = 5.5452f /* 8 ln 2 */, kLog2e = 1.4426950408889634f;

ERI_DEBUG_BOUNDS_DEFINE(fa_bias)

// z[i] = s[i] * scale + bias[k0 + i] for 32 keys; keys at or beyond Lk are -inf. In natural units, not in those of exp2:
// a mask of the type's lowest value is finite, and times log2(e) it would not be.
__device__ __forceinline__ void biased32(const BiasParams& p, const void* brow, int k0, const uint32_t (&r)[32], float (&z)[32]) {
  if (p.vec && k0 + 32 <= p.Lk) {
    const bf16x8* b8 = reinterpret_cast<const bf16x8*>(static_cast<const bf16*>(brow) + k0);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float b[8];
      unpack8(b8[g], b);
#pragma unroll
      for (int i = 0; i < 8; ++i) z[g * 8 + i] = fmaf(__uint_as_float(r[g * 8 + i]), p.scale, b[i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float b = -INFINITY;
      if (k0 + i < p.Lk)
        b = p.is_bool ? (static_cast<const uint8_t*>(brow)[k0 + i] ? 0.f : -INFINITY)
                      : __bfloat162float(static_cast<const bf16*>(brow)[k0 + i]);
      z[i] = b == -INFINITY ? b : fmaf(__uint_as_float(r[i]), p.scale, b);
    }
  }
}

template <int DH>
__global__ void __launch_bounds__(320, DH == 64 ? 2 : 1)
fa_bias_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const BiasParams p) {
  constexpr int CHUNKS = DH / 64;
  constexpr int CHUNK_BYTES = 128 * 128, TILE_BYTES = CHUNK_BYTES * CHUNKS;
  constexpr uint32_t S_COL = 0, O_COL = 128, P3_COL = O_COL + DH, TMEM = DH == 64 ? 256 : 512;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + TILE_BYTES;
  uint8_t* sV = sK + TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + TILE_BYTES);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 2, *v_full = bars + 3, *v_empty = bars + 4, *s_full = bars + 5,
           *p_full = bars + 6, *o_done = bars + 7;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  float* xchg = reinterpret_cast<float*>(bars + 16);   // [2][128] row maximum, [2][128] row sum

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = blockIdx.x * BQ, h = blockIdx.y, b = blockIdx.z;
  const int nkv = (p.Lk + BKV - 1) / BKV;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 8; ++i) mbar_init(bars + i, bars + i == p_full ? 8 : 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, TILE_BYTES);
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) tma_load_3d(sQ + c * CHUNK_BYTES, &tmQ, q_full, h * DH + c * 64, q0, b);
      for (int j = 0; j < nkv; ++j) {
        const uint32_t par = (uint32_t)(j & 1);
        if (!mbar_wait(k_empty, par ^ 1)) { atomicExch(p.err, 51); break; }
        mbar_expect_tx(k_full, TILE_BYTES);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) tma_load_3d(sK + c * CHUNK_BYTES, &tmK, k_full, h * DH + c * 64, j * BKV, b);
        if (!mbar_wait(v_empty, par ^ 1)) { atomicExch(p.err, 52); break; }
        mbar_expect_tx(v_full, TILE_BYTES);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) tma_load_3d(sV + c * CHUNK_BYTES, &tmV, v_full, h * DH + c * 64, j * BKV, b);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc_bf16(BQ, BKV, 0, 0), idesc_o = umma_idesc_bf16(BQ, DH, 0, 1);
      const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK), aV = smem_u32(sV);
      bool ok = mbar_wait(q_full, 0);
      if (!ok) atomicExch(p.err, 53);
      for (int j = 0; j < nkv && ok; ++j) {
        const uint32_t par = (uint32_t)(j & 1);
        if (!mbar_wait(k_full, par)) { atomicExch(p.err, 54); break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
          const uint64_t dq = umma_desc_kmajor(aQ + c * CHUNK_BYTES, 128), dk = umma_desc_kmajor(aK + c * CHUNK_BYTES, 128);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_bf16(tmem_base + S_COL, dq + kk * 2, dk + kk * 2, idesc_s, (c | kk) != 0);
        }
        umma_commit(s_full);
        umma_commit(k_empty);
        if (!mbar_wait(p_full, par)) { atomicExch(p.err, 55); break; }
        if (!mbar_wait(v_full, par)) { atomicExch(p.err, 56); break; }
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk) {
          // 32 keys take the 32 columns that their scores had: 16 columns of first terms, then 16 of second ones
          const uint32_t pcol = tmem_base + S_COL + (kk >> 1) * 32 + (kk & 1) * 8;
          const uint64_t dv = umma_desc_mn128(aV + kk * 2048, CHUNK_BYTES);
          umma_bf16_ts(tmem_base + O_COL, pcol, dv, idesc_o, (j | kk) != 0);
          umma_bf16_ts(tmem_base + O_COL, pcol + 16, dv, idesc_o, true);
          umma_bf16_ts(tmem_base + O_COL, tmem_base + P3_COL + kk * 8, dv, idesc_o, true);
        }
        umma_commit(o_done);
        umma_commit(v_empty);
      }
    }
  } else {
    const int qd = warp & 3, half = (warp - 2) >> 2;
    const int r_in = qd * 32 + lane, row = q0 + r_in;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t s_col = S_COL + half * 64;
    // rows beyond the last query read the last one's bias (their result is not written)
    const long long boff = b * p.sb + h * p.sh + (long long)min(row, p.Lq - 1) * p.sq;
    const void* brow = p.is_bool ? static_cast<const void*>(static_cast<const uint8_t*>(p.bias) + boff)
                                 : static_cast<const void*>(static_cast<const bf16*>(p.bias) + boff);
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nkv; ++j) {
      const uint32_t par = (uint32_t)(j & 1);
      if (ok && !mbar_wait(s_full, par)) {
        if (lane == 0) atomicExch(p.err, 57);
        ok = false;
      }
      if (!ok) {   // still meets its partners at the barrier and on p_full
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (lane == 0) mbar_arrive(p_full);
        continue;
      }
      tc_fence_after();
      const int kbase = j * BKV + half * 64;
      float mx = -INFINITY;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        float z[32];
        tmem_ld32(lane_addr + s_col + c * 32, r);
        tmem_ld_wait();
        biased32(p, brow, kbase + c * 32, r, z);
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, z[i]);
      }
      xchg[half * 128 + r_in] = mx;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      // (xchg needs no second barrier: the next tile's s_full waits for all eight warps' p_full)
      const float m_new = fmaxf(mx, xchg[(half ^ 1) * 128 + r_in]);
      if (j == 0) {
        m_used = m_new;
      } else {
        // (a row without a visible key so far has -inf on both sides: the difference is not a number, no rescale)
        const bool need = (m_new - m_used) > kRescaleThreshold;
        if (__any_sync(0xffffffffu, need)) {
          // s_full of this tile was committed after the products of the previous one: O is complete
          const float m_t = need ? m_new : m_used;
          const float alpha = need ? exp2f((m_used - m_t) * kLog2e) : 1.f;
#pragma unroll 1
          for (int c = 0; c < DH / 64; ++c) {
            uint32_t r[32];
            const uint32_t oc = O_COL + half * (DH / 2) + c * 32;
            tmem_ld32(lane_addr + oc, r);
            tmem_ld_wait();
            uint32_t a0[16], a1[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              a0[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              a1[i] = __float_as_uint(__uint_as_float(r[16 + i]) * alpha);
            }
            tmem_st16(lane_addr + oc, a0);
            tmem_st16(lane_addr + oc + 16, a1);
          }
          tmem_st_wait();
          l *= alpha;
          m_used = m_t;
        }
      }
      const float m_sub = m_used == -INFINITY ? 0.f : m_used;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        float z[32];
        tmem_ld32(lane_addr + s_col + c * 32, r);
        tmem_ld_wait();
        biased32(p, brow, kbase + c * 32, r, z);
        uint32_t p1[16], p2[16], p3[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float a = ex2_mufu((z[2 * i] - m_sub) * kLog2e), b = ex2_mufu((z[2 * i + 1] - m_sub) * kLog2e);
          l += a + b;
          p1[i] = pack_bf162(a, b);
          const float2 f = bf162_bits_to_float2(p1[i]);
          const float a2 = a - f.x, b2 = b - f.y;      // exact, as are the remainders of the remainders
          p2[i] = pack_bf162(a2, b2);
          const float2 t = bf162_bits_to_float2(p2[i]);
          p3[i] = pack_bf162(a2 - t.x, b2 - t.y);
        }
        tmem_st16(lane_addr + s_col + c * 32, p1);
        tmem_st16(lane_addr + s_col + c * 32 + 16, p2);
        tmem_st16(lane_addr + P3_COL + half * 32 + c * 16, p3);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok && !mbar_wait(o_done, (uint32_t)((nkv - 1) & 1))) {
      if (lane == 0) atomicExch(p.err, 58);
      ok = false;
    }
    xchg[256 + half * 128 + r_in] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l += xchg[256 + (half ^ 1) * 128 + r_in];
    if (ok) {
      tc_fence_after();
      const float inv_l = l == 0.f ? 0.f : 1.f / l;     // no visible key: zeros
      bf16* orow = p.out + (((size_t)b * p.Lq + row) * p.H + h) * DH + half * (DH / 2);
#pragma unroll 1
      for (int c = 0; c < DH / 64; ++c) {
        uint32_t r[32];
        tmem_ld32(lane_addr + O_COL + half * (DH / 2) + c * 32, r);
        tmem_ld_wait();
        if (row < p.Lq) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[g * 8 + i]) * inv_l;
            if (ERI_DBG_RANGE(p.out, (size_t)p.B * p.Lq * p.H * DH * 2, orow + c * 32 + g * 8, 16, 53))
              *reinterpret_cast<bf16x8*>(orow + c * 32 + g * 8) = pack8(v);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, TMEM);
  }
}

int* g_bias_err[64] = {nullptr};   // one error word per device

int make_map(CUtensorMap* m, const void* ptr, int B, int L, int H, int DH, long long ld) {
  uint64_t dims[3] = {(uint64_t)H * DH, (uint64_t)L, (uint64_t)B};
  uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)L * ld * 2};
  uint32_t box[3] = {64, 128, 1};
  return make_tensor_map(m, ptr, 3, dims, strides, box, 128);
}

template <int DH>
int launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const BiasParams& p, int dev, cudaStream_t st) {
  constexpr int SMEM = 3 * 128 * 128 * (DH / 64) + 1024 + 128 + 2048;
  static bool configured[64] = {};
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(fa_bias_fwd_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  fa_bias_fwd_kernel<DH><<<dim3((p.Lq + BQ - 1) / BQ, p.H, p.B), 320, SMEM, st>>>(q, k, v, p);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

int eri_fa_bias_check_error() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !g_bias_err[dev]) return 0;
  int h = 0;
  cudaMemcpy(&h, g_bias_err[dev], sizeof(int), cudaMemcpyDeviceToHost);
  if (h) cudaMemset(g_bias_err[dev], 0, sizeof(int));
  return h;
}

// q [B, Lq, H, DH], k / v [B, Lk, H, DH] with the token strides of ld; out contiguous. bias: bf16 or (is_bool) one byte
// per element, strides sb, sh, sq in elements (0 where it is broadcast), keys consecutive.
int eri_flash_attn_bias_fwd(const void* q, const void* k, const void* v, void* out, const void* bias, long long sb, long long sh,
                            long long sq, int is_bool, int B, int H, int Lq, int Lk, int DH, float scale,
                            const EriAttnStrides* ld, void* stream) {
  if (DH != 64 && DH != 128) return -1;
  EriAttnStrides s = *ld;
  for (long long* t : {&s.q, &s.k, &s.v}) {
    if (*t == 0) *t = (long long)H * DH;
    if (*t < (long long)H * DH || *t % 8) return -7;
  }
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) return -7;
  if (Lq < 1 || Lk < 1) return -2;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  if (!g_bias_err[dev]) {
    if (cudaMalloc(&g_bias_err[dev], sizeof(int)) != cudaSuccess) return -3;
    cudaMemset(g_bias_err[dev], 0, sizeof(int));
  }
  CUtensorMap tq, tk, tv;
  if (make_map(&tq, q, B, Lq, H, DH, s.q) || make_map(&tk, k, B, Lk, H, DH, s.k) || make_map(&tv, v, B, Lk, H, DH, s.v)) return -4;
  BiasParams p;
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk;
  p.scale = scale;
  p.out = (bf16*)out; p.bias = bias; p.sb = sb; p.sh = sh; p.sq = sq; p.is_bool = is_bool; p.err = g_bias_err[dev];
  p.vec = !is_bool && sb % 8 == 0 && sh % 8 == 0 && sq % 8 == 0 && ((uintptr_t)bias & 15) == 0;
  cudaStream_t st = (cudaStream_t)stream;
  return DH == 128 ? launch<128>(tq, tk, tv, p, dev, st) : launch<64>(tq, tk, tv, p, dev, st);
}

}  // extern "C"

ERI_DEBUG_BOUNDS_EXPORT(fa_bias)
