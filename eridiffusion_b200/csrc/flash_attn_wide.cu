// Flash attention forward at head size 512 (the single-head spatial attention in the middle of the image
// autoencoders: 16384 tokens at 1024 x 1024), bf16 in / bf16 out, fp32 softmax state, no mask.
//
// One CTA per (128-query tile, half of the value columns, head, batch). The 512 output columns of a query tile do
// not fit into tensor memory next to the scores, so the two halves recompute S = Q K^T: 1.5 times the operations of
// a kernel that could hold them, against none of its traffic. TMEM: O 256 columns, S / P twice 128 columns, so that
// the next tile's QK^T runs under this tile's exponentials (shared memory holds one CTA per SM).
//   warp 0     TMA loads: Q once (8 chunks of 64 channels, 128 KB), then a ring of six 16 KB stages that carries, in
//              the order the products need them, K chunks (128 keys x 64 channels) and V slices (32 keys x 256
//              columns)
//   warp 1     tcgen05.mma issue: S(j+1), then O += P(j) V(j)  (P from TMEM, V as an MN-major operand)
//   warps 2-9  softmax, two threads per query row, as in flash_attn.cu (lazy rescale of O by more than 2^8)
// What bounds it: shared-memory bandwidth next to the tensor pipe. Per 128 keys: 3072 cycles of MMA, 4096 cycles of
// shared-memory fill and operand reads.
// Measured at 16384 tokens: the library's memory-efficient kernel 3660 us (0.15 PFLOP/s); with this one a 1024 x 1024
// decode takes 13.98 instead of 16.76 ms.
#include "attn_args.h"
#include "ptx.cuh"
#include "tma_host.h"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

struct WideParams {
  int B, H, Lq, Lk;
  float scale_log2;
  bf16* out;             // [B, Lq, H, 512], consecutive tokens out_ld elements apart
  long long out_ld;
  int* err;
};

constexpr int DH = 512, DV = 256, BQ = 128, BKV = 128;
constexpr int kChunk = 128 * 128;         // 128 rows x 64 bf16
constexpr int kStages = 6, kQChunks = DH / 64, kVSlices = BKV / 32;
constexpr int kSmem = (kQChunks + kStages) * kChunk + 1024 + 256 + 1024;
constexpr float kRescaleThreshold = 8.0f;  // log2 units
constexpr uint32_t O_COL = 0, S_COL = 256;

ERI_DEBUG_BOUNDS_DEFINE(fa_wide)

__global__ void __launch_bounds__(320, 1)
fa_wide_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const WideParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* ring = smem + kQChunks * kChunk;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + kStages * kChunk);
  uint64_t* full = bars;                    // [kStages]
  uint64_t* empty = bars + kStages;         // [kStages]
  uint64_t* q_full = bars + 2 * kStages;
  uint64_t* s_full = q_full + 1;            // [2]
  uint64_t* p_full = s_full + 2;            // [2]
  uint64_t* o_done = p_full + 2;            // [2]: a waiter may be two products behind, which one parity bit cannot tell
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  float* xchg = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);   // [2][128] row max / row sum exchange

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the two halves of a query tile are neighbours, so that they read the same K tiles at about the same time
  const int q0 = (blockIdx.x >> 1) * BQ, vh = blockIdx.x & 1, h = blockIdx.y, b = blockIdx.z;
  const int nkv = (p.Lk + BKV - 1) / BKV;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 8);
      mbar_init(&o_done[i], 1);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, kQChunks * kChunk);
#pragma unroll 1
      for (int c = 0; c < kQChunks; ++c) tma_load_3d(sQ + c * kChunk, &tmQ, q_full, h * DH + c * 64, q0, b);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      auto slot = [&]() -> uint8_t* {
        if (!mbar_wait(&empty[stage], phase ^ 1)) {
          atomicExch(p.err, 31);
          ok = false;
          return nullptr;
        }
        mbar_expect_tx(&full[stage], kChunk);
        return ring + stage * kChunk;
      };
      auto next = [&]() {
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      };
      // order of the products: S(0), then S(j + 1), PV(j)
      for (int j = -1; j < nkv && ok; ++j) {
        if (j + 1 < nkv)
          for (int c = 0; c < kQChunks && ok; ++c) {
            uint8_t* d = slot();
            if (!ok) break;
            tma_load_3d(d, &tmK, &full[stage], h * DH + c * 64, (j + 1) * BKV, b);
            next();
          }
        if (j >= 0)
          for (int s = 0; s < kVSlices && ok; ++s) {
            uint8_t* d = slot();
            if (!ok) break;
#pragma unroll
            for (int c = 0; c < DV / 64; ++c)
              tma_load_3d(d + c * 4096, &tmV, &full[stage], h * DH + vh * DV + c * 64, j * BKV + s * 32, b);
            next();
          }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc_bf16(BQ, BKV, 0, 0);
      const uint32_t idesc_o = umma_idesc_bf16(BQ, DV, 0, 1);   // V is MN-major
      const uint32_t aQ = smem_u32(sQ), aR = smem_u32(ring);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = mbar_wait(q_full, 0);
      if (!ok) atomicExch(p.err, 32);
      auto wait_stage = [&]() {
        if (!mbar_wait(&full[stage], phase)) {
          atomicExch(p.err, 33);
          ok = false;
        }
        tc_fence_after();
      };
      auto release = [&]() {
        umma_commit(&empty[stage]);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      };
      for (int j = -1; j < nkv && ok; ++j) {
        if (j + 1 < nkv) {
          // S(j + 1) overwrites P(j - 1): that product was issued before this one, and the pipe keeps their order
          const int buf = (j + 1) & 1;
          for (int c = 0; c < kQChunks && ok; ++c) {
            wait_stage();
            if (!ok) break;
            const uint64_t dq = umma_desc_kmajor(aQ + c * kChunk, 128);
            const uint64_t dk = umma_desc_kmajor(aR + stage * kChunk, 128);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem_base + S_COL + buf * 128, dq + kk * 2, dk + kk * 2, idesc_s, (c | kk) != 0);
            release();
          }
          if (ok) umma_commit(&s_full[buf]);
        }
        if (j >= 0 && ok) {
          const int buf = j & 1;
          if (!mbar_wait(&p_full[buf], (uint32_t)((j >> 1) & 1))) {
            atomicExch(p.err, 34);
            break;
          }
          tc_fence_after();
          for (int s = 0; s < kVSlices && ok; ++s) {
            wait_stage();
            if (!ok) break;
#pragma unroll
            for (int k2 = 0; k2 < 2; ++k2) {
              const int kk = s * 2 + k2;      // 16 keys each
              umma_bf16_ts(tmem_base + O_COL, tmem_base + S_COL + buf * 128 + (kk >> 2) * 64 + (kk & 3) * 8,
                           umma_desc_mn128(aR + stage * kChunk + k2 * 2048, 4096), idesc_o, (j | kk) != 0);
            }
            release();
          }
          if (ok) umma_commit(&o_done[buf]);
        }
      }
    }
  } else {
    // Warps w and w + 4 own the same 32 query rows and take 64 of a tile's 128 keys each; at the end, and when O is
    // rescaled, 128 of its 256 columns each.
    const int qd = warp & 3, half = (warp - 2) >> 2;
    const int r_in = qd * 32 + lane, row = q0 + r_in;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nkv; ++j) {
      const int buf = j & 1;
      const uint32_t s_col = S_COL + buf * 128 + half * 64;
      if (ok && !mbar_wait(&s_full[buf], (uint32_t)((j >> 1) & 1))) {
        if (lane == 0) atomicExch(p.err, 35);
        ok = false;
      }
      if (!ok) {
        // a warp that gave up still meets its partners at the barriers, so that none waits without a limit
        asm volatile("bar.sync 1, 256;" ::: "memory");
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (lane == 0) mbar_arrive(&p_full[buf]);
        continue;
      }
      tc_fence_after();
      const int kv_left = p.Lk - j * BKV - half * 64;
      const bool full_half = kv_left >= 64;
      float mx = -INFINITY;
      if (full_half) {
        uint32_t r[32], r2[32];
        tmem_ld32(lane_addr + s_col, r);
        tmem_ld32(lane_addr + s_col + 32, r2);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          mx = fmax3(mx, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
          mx = fmax3(mx, __uint_as_float(r2[i]), __uint_as_float(r2[i + 1]));
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t r[32];
          tmem_ld32(lane_addr + s_col + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i < kv_left) mx = fmaxf(mx, __uint_as_float(r[i]));
        }
      }
      xchg[half * 128 + r_in] = mx;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      mx = fmaxf(mx, xchg[(half ^ 1) * 128 + r_in]);
      // the next tile's scores may be ready already: nobody writes its maximum before all have read this tile's
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const float m_new = mx * p.scale_log2;
      if (j == 0) {
        m_used = m_new;
      } else {
        const bool need = (m_new - m_used) > kRescaleThreshold;
        if (__any_sync(0xffffffffu, need)) {
          // O must be complete up to the previous tile
          if (!mbar_wait(&o_done[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1))) {
            if (lane == 0) atomicExch(p.err, 36);
            ok = false;
            if (lane == 0) mbar_arrive(&p_full[buf]);
            continue;
          }
          tc_fence_after();
          const float m_t = need ? m_new : m_used;
          const float alpha = exp2f(m_used - m_t);
#pragma unroll 1
          for (int c = 0; c < DV / 64; ++c) {
            uint32_t r[32];
            const uint32_t oc = O_COL + half * (DV / 2) + c * 32;
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
      float lsum = 0.f;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld32(lane_addr + s_col + c * 32, r);
        tmem_ld_wait();
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float p0 = ex2_mufu(fmaf(__uint_as_float(r[2 * i]), p.scale_log2, -m_used));
          float p1 = ex2_mufu(fmaf(__uint_as_float(r[2 * i + 1]), p.scale_log2, -m_used));
          if (!full_half) {
            if (c * 32 + 2 * i >= kv_left) p0 = 0.f;
            if (c * 32 + 2 * i + 1 >= kv_left) p1 = 0.f;
          }
          lsum += p0 + p1;
          pk[i] = pack_bf162(p0, p1);
        }
        tmem_st16(lane_addr + s_col + c * 16, pk);
      }
      l += lsum;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[buf]);
    }
    if (ok && !mbar_wait(&o_done[(nkv - 1) & 1], (uint32_t)(((nkv - 1) >> 1) & 1))) {
      if (lane == 0) atomicExch(p.err, 37);
      ok = false;
    }
    xchg[half * 128 + r_in] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l += xchg[(half ^ 1) * 128 + r_in];
    if (ok) {
      tc_fence_after();
      const float inv_l = 1.f / l;
      bf16* orow = p.out + ((size_t)b * p.Lq + row) * p.out_ld + h * DH + vh * DV + half * (DV / 2);
#pragma unroll 1
      for (int c = 0; c < DV / 64; ++c) {
        uint32_t r[32];
        tmem_ld32(lane_addr + O_COL + half * (DV / 2) + c * 32, r);
        tmem_ld_wait();
        if (row < p.Lq) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[g * 8 + i]) * inv_l;
            if (ERI_DBG_RANGE(p.out, (((size_t)p.B * p.Lq - 1) * p.out_ld + (size_t)p.H * DH) * 2, orow + c * 32 + g * 8, 16, 52))
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
    tmem_dealloc(tmem_base, 512);
  }
}

int* g_wide_err[64] = {nullptr};   // one error word per device

int make_map(CUtensorMap* m, const void* ptr, int B, int L, int H, long long ld, uint32_t rows) {
  uint64_t dims[3] = {(uint64_t)H * DH, (uint64_t)L, (uint64_t)B};
  uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)L * ld * 2};
  uint32_t box[3] = {64, rows, 1};
  return make_tensor_map(m, ptr, 3, dims, strides, box, 128);
}

}  // namespace

extern "C" {

int eri_fa_wide_check_error() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !g_wide_err[dev]) return 0;
  int h = 0;
  cudaMemcpy(&h, g_wide_err[dev], sizeof(int), cudaMemcpyDeviceToHost);
  if (h) cudaMemset(g_wide_err[dev], 0, sizeof(int));
  return h;
}

// q [B, Lq, H, 512], k / v [B, Lk, H, 512], out [B, Lq, H, 512]; token strides in ld (attn_args.h). Lq, Lk >= 128 (a
// tile is 128 rows high).
int eri_flash_attn_wide_fwd(const void* q, const void* k, const void* v, void* out, int B, int H, int Lq, int Lk, float scale,
                            const EriAttnStrides* ld, void* stream) {
  EriAttnStrides s = *ld;
  for (long long* t : {&s.q, &s.k, &s.v, &s.out}) {
    if (*t == 0) *t = (long long)H * DH;
    if (*t < (long long)H * DH || *t % 8) return -7;
  }
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) return -7;
  if (Lq < 128 || Lk < 128) return -2;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  static bool configured[64] = {};
  if (!configured[dev]) {
    if (!g_wide_err[dev]) {
      if (cudaMalloc(&g_wide_err[dev], sizeof(int)) != cudaSuccess) return -3;
      cudaMemset(g_wide_err[dev], 0, sizeof(int));
    }
    if (cudaFuncSetAttribute(fa_wide_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  CUtensorMap tq, tk, tv;
  if (make_map(&tq, q, B, Lq, H, s.q, 128) || make_map(&tk, k, B, Lk, H, s.k, 128) || make_map(&tv, v, B, Lk, H, s.v, 32)) return -4;
  WideParams p;
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.out = (bf16*)out; p.out_ld = s.out; p.err = g_wide_err[dev];
  fa_wide_fwd_kernel<<<dim3(2 * ((Lq + BQ - 1) / BQ), H, B), 320, kSmem, (cudaStream_t)stream>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

}  // extern "C"

ERI_DEBUG_BOUNDS_EXPORT(fa_wide)
