// GEMM for products of few output tiles (a few hundred to a few thousand rows): out = epilogue(A op(B)) with the same
// plain epilogue family as gemm.cu (bias, GELU / SiLU + saved pre-activation, activation backward, gate + residual,
// LoRA K step) and all four operand majors.
//
// What bounds such a product on the persistent kernels: 12-160 tiles of 128 x 128 leave most SMs idle or make a second,
// nearly empty round, a tile's K steps are one serial chain (0.26 us per step: an SM takes in about 64 bytes of
// operands per cycle), and the prologue, the epilogue and its row-per-thread stores (5 us together) are exposed because
// a CTA owns its SM alone. Here
//   * the K range of a tile is split over a cluster of 1, 2, 4 or 8 CTAs; the fp32 partial tiles meet in distributed
//     shared memory and are added in split order (deterministic), each CTA finishing its share of the rows;
//   * two CTAs share an SM (three stages of operands each) when there are more CTAs than SMs, so that one's prologue
//     and epilogue run under the other's products;
//   * the epilogue goes through shared memory: 16 lanes write 256 consecutive bytes of an output row.
// Measured: see split_for().
// Roles: warp 0 TMA, warp 1 UMMA issue, warps 2-9 TMEM -> shared memory; the final sum and the epilogue use all warps.
#include "gemm_args.h"
#include "ptx.cuh"
#include "tma_host.h"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

struct FewParams {
  int M, N, num_k, splits, num_m;
  int lora_r, act, ldc, ld_pre, ldr, rows_per_batch, gate_stride;
  int a_mn, b_mn;
  float alpha;
  const bf16 *bias, *residual, *gate, *pre_in;
  bf16 *out, *pre_out;
  int* err;
  long long dbg_out_bytes, dbg_pre_bytes;   // debug build only
};

ERI_DEBUG_BOUNDS_DEFINE(gemm_few)

constexpr int BM = 128, BN = 128, BK = 64, kThreads = 320;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int PITCH = BN + 4;   // floats per row of a partial tile: 16-byte accesses of 8 rows hit 8 bank groups

__device__ __forceinline__ float act_of(float v, int act) { return act == 1 ? gelu_tanh_f(v) : silu_f(v); }
__device__ __forceinline__ float act_grad_of(float v, int act) { return act == 3 ? gelu_tanh_grad_f(v) : silu_grad_f(v); }

template <int STAGES>
__global__ void __launch_bounds__(kThreads, STAGES <= 3 ? 2 : 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
                const __grid_constant__ FewParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.splits > 1 ? (int)cluster_ctarank() : 0;     // cluster = (splits, 1, 1)
  const int tile = blockIdx.x / p.splits;
  const int m0 = (tile % p.num_m) * BM, n0 = (tile / p.num_m) * BN;   // the row tiles of one weight tile are neighbours
  const int k0 = (int)((long long)p.num_k * split / p.splits), k1 = (int)((long long)p.num_k * (split + 1) / p.splits);
  const bool lora = p.lora_r > 0 && split == p.splits - 1;
  const int steps = k1 - k0 + (lora ? 1 : 0);                      // at least one: num_k >= splits

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait(&empty[stage], phase ^ 1)) {
          atomicExch(p.err, 41);
          break;
        }
        uint8_t* sA = smem + stage * STAGE_BYTES;
        uint8_t* sB = sA + A_BYTES;
        if (k0 + i < k1) {
          const int k = (k0 + i) * BK;
          mbar_expect_tx(&full[stage], STAGE_BYTES);
          if (!p.a_mn) {
            tma_load_2d(sA, &tmA, &full[stage], k, m0);
          } else {
            tma_load_2d(sA, &tmA, &full[stage], m0, k);
            tma_load_2d(sA + BK * 128, &tmA, &full[stage], m0 + 64, k);
          }
          if (!p.b_mn) {
            tma_load_2d(sB, &tmB, &full[stage], k, n0);
          } else {
            tma_load_2d(sB, &tmB, &full[stage], n0, k);
            tma_load_2d(sB + BK * 128, &tmB, &full[stage], n0 + 64, k);
          }
        } else {
          // lora_h may still be in production by the previous kernel (dependent launch)
          griddep_wait();
          mbar_expect_tx(&full[stage], (BM + BN) * p.lora_r * 2);
          tma_load_2d(sA, &tmA2, &full[stage], 0, m0);
          tma_load_2d(sB, &tmB2, &full[stage], 0, n0);
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(BM, BN, p.a_mn, p.b_mn), idesc_lora = umma_idesc_bf16(BM, BN, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait(&full[stage], phase)) {
          atomicExch(p.err, 42);
          ok = false;
          // the copies behind this one may still be on their way into this CTA's shared memory
          for (int s = 1; s < STAGES && i + s < steps; ++s) {
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1;
            }
            mbar_wait(&full[stage], phase);
          }
          break;
        }
        tc_fence_after();
        const uint32_t sA = smem_u32(smem + stage * STAGE_BYTES), sB = sA + A_BYTES;
        if (k0 + i < k1) {
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            const uint64_t da = p.a_mn ? umma_desc_mn128(sA + kk * 2048, BK * 128) : umma_desc_kmajor(sA, 128) + kk * 2;
            const uint64_t db = p.b_mn ? umma_desc_mn128(sB + kk * 2048, BK * 128) : umma_desc_kmajor(sB, 128) + kk * 2;
            umma_bf16(tmem_base, da, db, idesc, (i | kk) != 0);
          }
        } else {
          const uint64_t da = umma_desc_kmajor(sA, p.lora_r * 2), db = umma_desc_kmajor(sB, p.lora_r * 2);
          for (int kk = 0; kk < p.lora_r / 16; ++kk) umma_bf16(tmem_base, da + kk * 2, db + kk * 2, idesc_lora, (i | kk) != 0);
        }
        umma_commit(&empty[stage]);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) umma_commit(acc_full);
    }
  } else {
    // this CTA's partial tile -> shared memory (the stages are free: the commit behind acc_full covers every product
    // that read them)
    const int q = warp & 3, half = (warp - 2) >> 2;
    const bool ok = mbar_wait(acc_full, 0);
    if (!ok && lane == 0) atomicExch(p.err, 43);
    tc_fence_after();
    float* row = reinterpret_cast<float*>(smem) + (q * 32 + lane) * PITCH + half * 64;
    if (ok) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + half * 64 + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<uint4*>(row + c * 32 + i * 4) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
      }
    } else {
      // the tile becomes NaN, never what the shared memory happened to hold
      for (int i = 0; i < 64; ++i) row[i] = __int_as_float(0x7fffffff);
    }
    tc_fence_before();
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync_all(); else __syncthreads();
  tc_fence_after();

  // rows [r_lo, r_lo + band) of the tile are this CTA's to finish; an item is eight columns of a row
  const int band = BM / p.splits, r_lo = split * band;
  const uint32_t part = smem_u32(smem);
  for (int it = threadIdx.x; it < band * (BN / 8); it += kThreads) {
    const int rl = r_lo + it / (BN / 8), c = (it % (BN / 8)) * 8, row = m0 + rl, col = n0 + c;
    if (row >= p.M || col >= p.N) continue;
    float v[8];
    const uint32_t off = part + (uint32_t)(rl * PITCH + c) * 4u;
    if (p.splits == 1) {
      const float4* s = reinterpret_cast<const float4*>(smem + (size_t)(rl * PITCH + c) * 4);
      const float4 lo = s[0], hi = s[1];
      v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll 4
      for (int s = 0; s < p.splits; ++s) {
        const uint32_t src = map_to_cta(off, (uint32_t)s);
        const float4 lo = ld_shared_cluster_v4(src), hi = ld_shared_cluster_v4(src + 16);
        v[0] += lo.x; v[1] += lo.y; v[2] += lo.z; v[3] += lo.w;
        v[4] += hi.x; v[5] += hi.y; v[6] += hi.z; v[7] += hi.w;
      }
    }
    float t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= p.alpha;
    if (p.bias) {
      unpack8(*reinterpret_cast<const bf16x8*>(p.bias + col), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += t[j];
    }
    if (p.act == 1 || p.act == 2) {
      if (p.pre_out && ERI_DBG_RANGE(p.pre_out, p.dbg_pre_bytes, p.pre_out + (size_t)row * p.ld_pre + col, 16, 84))
        *reinterpret_cast<bf16x8*>(p.pre_out + (size_t)row * p.ld_pre + col) = pack8(v);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = act_of(v[j], p.act);
    } else if (p.act == 3 || p.act == 4) {
      unpack8(*reinterpret_cast<const bf16x8*>(p.pre_in + (size_t)row * p.ld_pre + col), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= act_grad_of(t[j], p.act);
    }
    if (p.gate) {
      unpack8(*reinterpret_cast<const bf16x8*>(p.gate + (size_t)(row / p.rows_per_batch) * p.gate_stride + col), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= t[j];
    }
    if (p.residual) {
      unpack8(*reinterpret_cast<const bf16x8*>(p.residual + (size_t)row * p.ldr + col), t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += t[j];
    }
    bf16* o = p.out + (size_t)row * p.ldc + col;
    if (ERI_DBG_RANGE(p.out, p.dbg_out_bytes, o, 16, 83)) *reinterpret_cast<bf16x8*>(o) = pack8(v);
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync_all();   // no CTA leaves (and frees its shared memory) while a peer may read its partial
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, BN);
  }
}

template <int STAGES>
int launch(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& a2, const CUtensorMap& b2, const FewParams& p, int tiles,
           bool pdl, int dev, cudaStream_t st) {
  constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;
  static bool configured[64] = {};
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (p.splits > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = p.splits; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return (int)cudaLaunchKernelEx(&cfg, gemm_few_kernel<STAGES>, a, b, a2, b2, p);
}

struct FewState {
  int* err = nullptr;
  int sms = 0;
};
FewState g_few[64];

// Splits of the K range for `tiles` tiles of `num_k` steps (0: the persistent kernels are faster). Two CTAs on one SM
// only help while the prologue and the epilogue are a good part of a tile, since they share the SM's operand intake; a
// split pays while it brings in SMs that would idle and leaves every CTA eight steps. [M x N x K], us, this kernel
// against the persistent ones (cold weights):
//   one split, tiles <= 2 SMs  4096x640x640 9.8 / 12.4, 2048x1280x1280 13.7 / 15.5, 1024x3840x1280 14.6 / 16.4; but
//                              2048x1280x5120 35.4 / 32.9, 384x9216x3072 26.8 / 25.5
//   two splits, fit the SMs    384x3072x12288 31.5 / 48.0, 256x4096x10240 27.6 / 41.5, 256x4096x4096 15.9 / 20.7
//   two splits, more than SMs  1024x1280x1280 13.0 / 10.3 (one split: 10.2)
//   four / eight splits        320x512x2048 9.9 / 11.8 against 12.9
int split_for(int tiles, int num_k, int sms) {
  if (tiles > 2 * sms || (tiles > sms && num_k > 24)) return 0;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= sms && num_k >= 16 * s) s *= 2;
  return s;
}

}  // namespace

extern "C" {

int eri_gemm_few_check_error() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !g_few[dev].err) return 0;
  int h = 0;
  cudaMemcpy(&h, g_few[dev].err, sizeof(int), cudaMemcpyDeviceToHost);
  if (h) cudaMemset(g_few[dev].err, 0, sizeof(int));
  return h;
}

// Answers -30 where another kernel is the better or the only one. force_bn < 0: -force_bn splits (1, 2, 4 or 8).
int eri_gemm_few_bf16(const EriGemmArgs* g, void* stream) {
  if (g->n_split || g->out2 || g->n_copy || g->scatter_world || g->rowsq || g->glu || g->force_bn > 0 || g->b_local) return -30;
  if (g->M < BM || g->N < BN || g->K < BK || g->K % 8 || g->N % 8 || g->lda % 8 || g->ldb % 8 || g->ldc % 8) return -30;
  if (g->a_mn && g->M % 8) return -30;
  if (g->lora_r && g->lora_r != 16 && g->lora_r != 32 && g->lora_r != 64) return -30;
  // every epilogue operand is accessed in 16-byte words
  if (((uintptr_t)g->out | (uintptr_t)g->bias | (uintptr_t)g->residual | (uintptr_t)g->gate | (uintptr_t)g->pre_in |
       (uintptr_t)g->pre_out) & 15)
    return -30;
  if ((g->residual && g->ldr % 8) || ((g->pre_in || g->pre_out) && g->ld_pre % 8) || (g->gate && g->gate_stride % 8)) return -30;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -30;
  FewState& s = g_few[dev];
  cudaStream_t st = (cudaStream_t)stream;
  if (!s.err) {
    cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaMalloc(&s.err, sizeof(int)) != cudaSuccess) return -3;
    cudaMemset(s.err, 0, sizeof(int));
  }
  FewParams p = {};
  p.num_m = (g->M + BM - 1) / BM;
  const int tiles = p.num_m * ((g->N + BN - 1) / BN);
  p.num_k = (g->K + BK - 1) / BK;
  p.splits = g->force_bn < 0 ? -g->force_bn : split_for(tiles, p.num_k, s.sms);
  if (p.splits == 0) return -30;
  if ((p.splits & (p.splits - 1)) || p.splits > 8 || p.splits > p.num_k) return -16;
  p.M = g->M; p.N = g->N; p.lora_r = g->lora_r; p.act = g->act; p.ldc = g->ldc; p.ld_pre = g->ld_pre; p.ldr = g->ldr;
  p.rows_per_batch = g->rows_per_batch > 0 ? g->rows_per_batch : g->M;
  p.gate_stride = g->gate_stride; p.a_mn = g->a_mn; p.b_mn = g->b_mn; p.alpha = g->alpha;
  p.bias = (const bf16*)g->bias; p.residual = (const bf16*)g->residual; p.gate = (const bf16*)g->gate;
  p.pre_in = (const bf16*)g->pre_in; p.out = (bf16*)g->out; p.pre_out = (bf16*)g->pre_out; p.err = s.err;
  p.dbg_out_bytes = g->dbg_out_bytes; p.dbg_pre_bytes = g->dbg_pre_bytes;

  CUtensorMap ta, tb, ta2, tb2;
  auto operand = [](CUtensorMap* m, const void* ptr, int mn, int rows, int K, long long ld) {
    uint64_t d[2] = {(uint64_t)(mn ? rows : K), (uint64_t)(mn ? K : rows)};
    uint64_t sb[1] = {(uint64_t)ld * 2};
    uint32_t bx[2] = {64, mn ? (uint32_t)BK : 128u};
    return make_tensor_map(m, ptr, 2, d, sb, bx, 128);
  };
  if (operand(&ta, g->a, g->a_mn, g->M, g->K, g->lda)) return -20;
  if (operand(&tb, g->b, g->b_mn, g->N, g->K, g->ldb)) return -21;
  if (g->lora_r) {
    auto low = [&](CUtensorMap* m, const void* ptr, int rows, long long ld) {
      uint64_t d[2] = {(uint64_t)g->lora_r, (uint64_t)rows};
      uint64_t sb[1] = {(uint64_t)ld * 2};
      uint32_t bx[2] = {(uint32_t)g->lora_r, 128};
      return make_tensor_map(m, ptr, 2, d, sb, bx, g->lora_r * 2);
    };
    if (low(&ta2, g->lora_h, g->M, g->ld_h)) return -22;
    if (low(&tb2, g->lora_b, g->N, g->ld_lb)) return -23;
  } else {
    ta2 = ta;
    tb2 = tb;
  }
  const bool pdl = g->pdl && g->lora_r;
  return tiles * p.splits <= s.sms ? launch<6>(ta, tb, ta2, tb2, p, tiles, pdl, dev, st)
                                   : launch<3>(ta, tb, ta2, tb2, p, tiles, pdl, dev, st);
}

}  // extern "C"

ERI_DEBUG_BOUNDS_EXPORT(gemm_few)
