// GroupNorm (+ optional SiLU) for channels-last activations [N, HW, C], forward and backward.
//
// Each direction is two bandwidth-bound passes over the activation and nothing else:
//   column pass   per-channel sums over a chunk of rows, one partial record per (n, chunk):
//                 forward  (sum x, sum x^2) per group;  backward  (sum dz, sum dz * xhat) per channel and,
//                 weighted by w, per group;  dz = dy * act'(z)
//   apply pass    first adds the partial records of its sample (in chunk order: results do not depend on timing),
//                 then forward  y = act(x * a + c) with a = w * rstd, c = b - mean * a held in registers,
//                 backward dx = rstd * (dz * w - s1 - xhat * s2); the backward's last CTAs add the per-channel
//                 records into the parameter gradients instead.
// A thread owns eight fixed channels and walks over rows, so the per-channel constants are loaded once and every
// access is one 16-byte vector. What bounds it: DRAM (or L2) traffic of the activation, 2 reads + 1 write. The
// version before used float atomics for the sums and eleven elementwise launches on the [N, C] statistics
// between the passes: a 1280-channel 32 x 32 layer took 43 us forward, of which 9 us were the two passes.
// The reference's GroupNorm is a forward-only NCHW kernel with one warp-shuffle reduction per group
// (crates/core/src/cuda/kernels/group_norm.cu); its SDXL ResBlocks apply SiLU as a separate pass
// (crates/training/src/sdxl/runtime.rs).
#include "ptx.cuh"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

struct GnArgs {
  const bf16 *x, *dy, *w, *b;
  float *mean, *rstd;        // [N, G]
  float* part;               // [N, chunks, G, 2] group records
  float* part_c;             // [N, chunks, C, 2 or 3] channel records (backward; sum xhat last, with pre only)
  bf16 *out, *dw, *db;
  // x + pre_c[c] + pre_nc[n, c] is what gets normalised (either may be null): the bias of the convolution that
  // produced x and a per-sample embedding, added here instead of in passes of their own
  const bf16 *pre_c, *pre_nc;
  bf16 *dpre_c, *dpre_nc;    // their gradients: sums of dx
  int N, HW, C, G, silu, chunks, rows_per_chunk, accumulate, apply_ctas;
  int gchunks;               // group records per sample that the apply pass adds (1 after a fold)
  float eps;
};

// A thread per eight channels at least: 640 threads up to 5120 channels, 1024 (and half the registers) up to 8192.
constexpr int kUnroll = 4, kMaxThreads = 640, kWideThreads = 1024;
// Partial records an apply CTA adds itself; more are folded by a launch of their own, because every apply CTA
// re-reads all of them (64 records of 32 groups: 16 KB from L2, about a microsecond).
constexpr int kMaxDirectChunks = 64;

__device__ __forceinline__ float silu_of(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float silu_grad_of(float z) {
  const float s = 1.f / (1.f + __expf(-z));
  return s * (1.f + z * (1.f - s));
}

// Adds the group records of sample n in chunk order into smem s[2 * G].
__device__ __forceinline__ void fold_groups(const GnArgs& a, int n, float* s) {
  const float* p = a.part + (size_t)n * a.gchunks * a.G * 2;
  for (int i = threadIdx.x; i < 2 * a.G; i += blockDim.x) {
    float v = 0.f;
#pragma unroll 8
    for (int c = 0; c < a.gchunks; ++c) v += p[(size_t)c * a.G * 2 + i];
    s[i] = v;
  }
  __syncthreads();
}

// The per-channel addend of x for eight channels.
__device__ __forceinline__ void load_pre(const GnArgs& a, int n, int v, float (&pr)[8]) {
  float t[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) pr[j] = 0.f;
  if (a.pre_c) unpack8(reinterpret_cast<const bf16x8*>(a.pre_c)[v], pr);
  if (a.pre_nc) {
    unpack8(reinterpret_cast<const bf16x8*>(a.pre_nc + (size_t)n * a.C)[v], t);
#pragma unroll
    for (int j = 0; j < 8; ++j) pr[j] += t[j];
  }
}

template <bool BWD, bool PRE, int THREADS>
__global__ void __launch_bounds__(THREADS) gn_column_kernel(const GnArgs a) {
  constexpr int S = BWD && PRE ? 3 : 2;
  extern __shared__ float sm[];     // [R][C][S] partial sums of the CTA's row lanes
  const int n = blockIdx.y, nvec = a.C >> 3;
  const int R = blockDim.x / nvec;
  const int v = threadIdx.x % nvec, rr = threadIdx.x / nvec;
  const int r0 = blockIdx.x * a.rows_per_chunk, r1 = min(a.HW, r0 + a.rows_per_chunk);
  float s0[8], s1[8], s2[8], pr[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s0[j] = s1[j] = s2[j] = pr[j] = 0.f;
  if (PRE && rr < R) load_pre(a, n, v, pr);
  const bf16x8* xp = reinterpret_cast<const bf16x8*>(a.x + (size_t)n * a.HW * a.C) + v;
  if (rr < R) {
    if constexpr (!BWD) {
      for (int r = r0 + rr; r < r1; r += R * kUnroll) {
        bf16x8 q[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
          if (r + u * R < r1) q[u] = xp[(size_t)(r + u * R) * nvec];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
          if (r + u * R < r1) {
            float f[8];
            unpack8(q[u], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (PRE) f[j] += pr[j];
              s0[j] += f[j];
              s1[j] = fmaf(f[j], f[j], s1[j]);
            }
          }
      }
    } else {
      const bf16x8* gp = reinterpret_cast<const bf16x8*>(a.dy + (size_t)n * a.HW * a.C) + v;
      const int cpg = a.C / a.G;
      float wv[8], bv[8], mu[8], rs[8];
      unpack8(reinterpret_cast<const bf16x8*>(a.w)[v], wv);
      if (a.b) {
        unpack8(reinterpret_cast<const bf16x8*>(a.b)[v], bv);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) bv[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int g = (v * 8 + j) / cpg;
        mu[j] = a.mean[n * a.G + g] - pr[j];
        rs[j] = a.rstd[n * a.G + g];
      }
      for (int r = r0 + rr; r < r1; r += R * 2) {
        bf16x8 q[2], d[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (r + u * R < r1) {
            q[u] = xp[(size_t)(r + u * R) * nvec];
            d[u] = gp[(size_t)(r + u * R) * nvec];
          }
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (r + u * R < r1) {
            float f[8], g[8];
            unpack8(q[u], f);
            unpack8(d[u], g);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float xh = (f[j] - mu[j]) * rs[j];
              const float dz = a.silu ? g[j] * silu_grad_of(fmaf(xh, wv[j], bv[j])) : g[j];
              s0[j] += dz;
              s1[j] = fmaf(dz, xh, s1[j]);
              if (PRE) s2[j] += xh;
            }
          }
      }
    }
    float* o = sm + ((size_t)rr * a.C + v * 8) * S;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[S * j] = s0[j];
      o[S * j + 1] = s1[j];
      if (S == 3) o[S * j + 2] = s2[j];
    }
  }
  __syncthreads();
  // row lanes -> one record per channel, in the first lane's slots
  for (int i = threadIdx.x; i < S * a.C; i += blockDim.x) {
    float t = sm[i];
    for (int r = 1; r < R; ++r) t += sm[(size_t)r * a.C * S + i];
    if constexpr (BWD) {
      a.part_c[((size_t)n * a.chunks + blockIdx.x) * a.C * S + i] = t;
      t *= __bfloat162float(a.w[i / S]);
    }
    sm[i] = t;
  }
  __syncthreads();
  const int cpg = a.C / a.G;
  float* dst = a.part + ((size_t)n * a.chunks + blockIdx.x) * a.G * 2;
  for (int i = threadIdx.x; i < 2 * a.G; i += blockDim.x) {
    const int g = i >> 1;
    float t = 0.f;
    for (int c = 0; c < cpg; ++c) t += sm[(g * cpg + c) * S + (i & 1)];
    dst[i] = t;
  }
}

// Many chunks: their group records folded into one (one CTA per sample; several lanes per record word, or with more than
// 512 groups several words per thread).
__global__ void gn_fold_kernel(GnArgs a, float* folded) {
  const int n = blockIdx.x, lanes = blockDim.x / (2 * a.G);
  extern __shared__ float sm[];     // [lanes][2 * G]
  if (lanes == 0) {
    for (int i = threadIdx.x; i < 2 * a.G; i += blockDim.x) {
      float v = 0.f;
      for (int c = 0; c < a.chunks; ++c) v += a.part[((size_t)n * a.chunks + c) * a.G * 2 + i];
      folded[(size_t)n * a.G * 2 + i] = v;
    }
    return;
  }
  const int i = threadIdx.x % (2 * a.G), l = threadIdx.x / (2 * a.G);
  const float* p = a.part + (size_t)n * a.chunks * a.G * 2;
  if (l < lanes) {
    float v = 0.f;
#pragma unroll 8
    for (int c = l; c < a.chunks; c += lanes) v += p[(size_t)c * a.G * 2 + i];
    sm[l * 2 * a.G + i] = v;
  }
  __syncthreads();
  if (l == 0) {
    float v = 0.f;
    for (int k = 0; k < lanes; ++k) v += sm[k * 2 * a.G + i];
    folded[(size_t)n * a.G * 2 + i] = v;
  }
}

// Parameter gradients of 32 channels: eight lanes per channel over the chunk records of every sample.
template <bool PRE>
__device__ __forceinline__ void param_gradients(const GnArgs& a, int cta, float* sm) {
  constexpr int S = PRE ? 3 : 2;
  const int lanes = blockDim.x / 32, cl = threadIdx.x & 31, l = threadIdx.x >> 5, c = cta * 32 + cl;
  const int cpg = a.C / a.G;
  const float inv_m = 1.f / ((float)a.HW * (float)cpg);
  float dw = 0.f, db = 0.f, dp = 0.f;
  for (int n = 0; n < a.N; ++n) {
    float t[3] = {0.f, 0.f, 0.f}, gs[2] = {0.f, 0.f};
    if (c < a.C) {
      for (int k = l; k < a.chunks; k += lanes) {
        const float* p = a.part_c + (((size_t)n * a.chunks + k) * a.C + c) * S;
#pragma unroll
        for (int i = 0; i < S; ++i) t[i] += p[i];
      }
      if (PRE)
        for (int k = l; k < a.gchunks; k += lanes) {
          const float* p = a.part + (((size_t)n * a.gchunks + k) * a.G + c / cpg) * 2;
          gs[0] += p[0];
          gs[1] += p[1];
        }
    }
    __syncthreads();
    float* mine = sm + (l * 32 + cl) * 5;
    mine[0] = t[0]; mine[1] = t[1]; mine[2] = t[2]; mine[3] = gs[0]; mine[4] = gs[1];
    __syncthreads();
    if (l == 0 && c < a.C) {
      float r[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
      for (int k = 0; k < lanes; ++k)
#pragma unroll
        for (int i = 0; i < 5; ++i) r[i] += sm[(k * 32 + cl) * 5 + i];
      db += r[0];
      dw += r[1];
      if (PRE) {
        // sum over the rows of dx = rstd * (dz * w - s1 - xhat * s2)
        const float d = a.rstd[n * a.G + c / cpg] * (__bfloat162float(a.w[c]) * r[0] - (float)a.HW * r[3] * inv_m - r[4] * inv_m * r[2]);
        dp += d;
        if (a.dpre_nc) a.dpre_nc[(size_t)n * a.C + c] = __float2bfloat16(d);
      }
    }
  }
  if (l == 0 && c < a.C) {
    if (a.dw) a.dw[c] = __float2bfloat16(dw + ((a.accumulate & 1) ? __bfloat162float(a.dw[c]) : 0.f));
    if (a.db) a.db[c] = __float2bfloat16(db + ((a.accumulate & 2) ? __bfloat162float(a.db[c]) : 0.f));
    if (a.dpre_c) a.dpre_c[c] = __float2bfloat16(dp + ((a.accumulate & 4) ? __bfloat162float(a.dpre_c[c]) : 0.f));
  }
}

template <bool BWD, bool PRE, int THREADS>
__global__ void __launch_bounds__(THREADS) gn_apply_kernel(const GnArgs a) {
  extern __shared__ float sm[];     // [2 * G]; parameter CTAs [threads / 32][32][5]
  const int nvec = a.C >> 3;
  if (BWD && (int)blockIdx.x >= a.apply_ctas) {
    if (blockIdx.y == 0) param_gradients<PRE>(a, blockIdx.x - a.apply_ctas, sm);
    return;
  }
  const int n = blockIdx.y, cpg = a.C / a.G;
  const float inv_m = 1.f / ((float)a.HW * (float)cpg);
  fold_groups(a, n, sm);
  if constexpr (!BWD) {
    for (int g = threadIdx.x; g < a.G; g += blockDim.x) {
      const float mean = sm[2 * g] * inv_m;
      const float var = sm[2 * g + 1] * inv_m - mean * mean;      // inf - inf where the squares overflow: stays NaN
      const float rstd = rsqrtf((var < 0.f ? 0.f : var) + a.eps);
      sm[2 * g] = mean;
      sm[2 * g + 1] = rstd;
      if (blockIdx.x == 0 && a.mean) {
        a.mean[n * a.G + g] = mean;
        a.rstd[n * a.G + g] = rstd;
      }
    }
    __syncthreads();
  }
  const int R = blockDim.x / nvec;
  const int v = threadIdx.x % nvec, rr = threadIdx.x / nvec;
  if (rr >= R) return;
  float wv[8], bv[8], pr[8];
  unpack8(reinterpret_cast<const bf16x8*>(a.w)[v], wv);
  if (a.b) {
    unpack8(reinterpret_cast<const bf16x8*>(a.b)[v], bv);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) bv[j] = 0.f;
  }
  if (PRE) load_pre(a, n, v, pr);
  const size_t base = (size_t)n * a.HW * nvec + v;
  const bf16x8* xp = reinterpret_cast<const bf16x8*>(a.x) + base;
  bf16x8* op = reinterpret_cast<bf16x8*>(a.out) + base;
  const int step = a.apply_ctas * R;
  if constexpr (!BWD) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int g = (v * 8 + j) / cpg;
      wv[j] *= sm[2 * g + 1];
      bv[j] = fmaf((PRE ? pr[j] : 0.f) - sm[2 * g], wv[j], bv[j]);
    }
    for (int r = blockIdx.x * R + rr; r < a.HW; r += step * kUnroll) {
      bf16x8 q[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        if (r + u * step < a.HW) q[u] = xp[(size_t)(r + u * step) * nvec];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        if (r + u * step < a.HW) {
          float f[8];
          unpack8(q[u], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float z = fmaf(f[j], wv[j], bv[j]);
            f[j] = a.silu ? silu_of(z) : z;
          }
          op[(size_t)(r + u * step) * nvec] = pack8(f);
        }
    }
  } else {
    const bf16x8* gp = reinterpret_cast<const bf16x8*>(a.dy) + base;
    float mu[8], rs[8], t1[8], t2[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int g = (v * 8 + j) / cpg;
      mu[j] = a.mean[n * a.G + g] - (PRE ? pr[j] : 0.f);
      rs[j] = a.rstd[n * a.G + g];
      t1[j] = sm[2 * g] * inv_m;
      t2[j] = sm[2 * g + 1] * inv_m;
    }
    for (int r = blockIdx.x * R + rr; r < a.HW; r += step * 2) {
      bf16x8 q[2], d[2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (r + u * step < a.HW) {
          q[u] = xp[(size_t)(r + u * step) * nvec];
          d[u] = gp[(size_t)(r + u * step) * nvec];
        }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (r + u * step < a.HW) {
          float f[8], g[8];
          unpack8(q[u], f);
          unpack8(d[u], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xh = (f[j] - mu[j]) * rs[j];
            const float dz = a.silu ? g[j] * silu_grad_of(fmaf(xh, wv[j], bv[j])) : g[j];
            f[j] = rs[j] * (dz * wv[j] - t1[j] - xh * t2[j]);
          }
          op[(size_t)(r + u * step) * nvec] = pack8(f);
        }
    }
  }
}

struct GnPlan {
  int threads, R, chunks, rows_per_chunk, apply_ctas;
};

// At least four rows per thread and about four column CTAs per SM; the apply pass about eight per SM.
GnPlan plan_for(int N, int HW, int C) {
  GnPlan p;
  const int nvec = C >> 3;
  p.R = 256 / nvec;
  if (p.R < 1) p.R = 1;
  p.threads = (p.R * nvec + 31) / 32 * 32;
  const int min_rows = p.R * kUnroll;
  int want = (148 * 4 + N - 1) / N;
  int rows = (HW + want - 1) / want;
  rows = (rows + min_rows - 1) / min_rows * min_rows;
  p.rows_per_chunk = rows;
  p.chunks = (HW + rows - 1) / rows;
  int ctas = (148 * 8 + N - 1) / N;
  const int most = (HW + p.R * 2 - 1) / (p.R * 2);
  p.apply_ctas = ctas < most ? ctas : most;
  return p;
}

template <bool BWD, bool PRE, int THREADS>
int run_v(GnArgs a, float* ws, cudaStream_t st) {
  const GnPlan p = plan_for(a.N, a.HW, a.C);
  a.chunks = a.gchunks = p.chunks;
  a.rows_per_chunk = p.rows_per_chunk;
  a.apply_ctas = p.apply_ctas;
  a.part = ws;
  float* folded = ws + (size_t)a.N * p.chunks * a.G * 2;
  a.part_c = folded + (size_t)a.N * a.G * 2;
  constexpr int S = BWD && PRE ? 3 : 2;
  const int smem = p.R * a.C * S * (int)sizeof(float);
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -2;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(gn_column_kernel<BWD, PRE, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             THREADS * 8 * S * (int)sizeof(float)) != cudaSuccess)
      return -2;
    configured[dev] = true;
  }
  gn_column_kernel<BWD, PRE, THREADS><<<dim3(p.chunks, a.N), p.threads, smem, st>>>(a);
  if (p.chunks > kMaxDirectChunks) {
    const int lanes = 1024 / (2 * a.G), threads = lanes ? lanes * 2 * a.G : 1024;
    gn_fold_kernel<<<a.N, threads, threads * sizeof(float), st>>>(a, folded);
    a.part = folded;
    a.gchunks = 1;
  }
  const bool params = BWD && (a.dw || a.db || a.dpre_c || a.dpre_nc);
  const int extra = params ? (a.C + 31) / 32 : 0;
  int smem_apply = 2 * a.G * (int)sizeof(float);
  if (params && p.threads * 5 * (int)sizeof(float) > smem_apply) smem_apply = p.threads * 5 * (int)sizeof(float);
  gn_apply_kernel<BWD, PRE, THREADS><<<dim3(p.apply_ctas + extra, a.N), p.threads, smem_apply, st>>>(a);
  return (int)cudaGetLastError();
}
template <bool BWD>
int run(const GnArgs& a, float* ws, cudaStream_t st) {
  const int threads = plan_for(a.N, a.HW, a.C).threads;
  if (threads > kWideThreads || a.G > 4096) return -1;
  const bool pre = a.pre_c || a.pre_nc;
  if (threads > kMaxThreads) return pre ? run_v<BWD, true, kWideThreads>(a, ws, st) : run_v<BWD, false, kWideThreads>(a, ws, st);
  return pre ? run_v<BWD, true, kMaxThreads>(a, ws, st) : run_v<BWD, false, kMaxThreads>(a, ws, st);
}

}  // namespace

extern "C" {

// fp32 words of workspace one call needs.
long long eri_gn_workspace(int N, int HW, int C, int G, int backward) {
  if (N < 1 || HW < 1 || C < 8) return 0;      // nothing to plan (the calls below refuse it)
  const GnPlan p = plan_for(N, HW, C);
  return (long long)N * (p.chunks + 1) * G * 2 + (backward ? (long long)N * p.chunks * C * 3 : 0);
}

// y = act(GroupNorm(x + pre_c + pre_nc)); mean / rstd [N, G] are written for the backward when given. pre_c [C] and
// pre_nc [N, C] (bf16) may be null.
int eri_gn_fwd(const void* x, const void* pre_c, const void* pre_nc, const void* w, const void* b, void* y, float* mean,
               float* rstd, float* ws, int N, int HW, int C, int G, float eps, int silu, void* stream) {
  if (N < 1 || HW < 1 || C < 8 || G < 1 || C % 8 || C % G) return -1;
  GnArgs a = {};
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.b = (const bf16*)b; a.out = (bf16*)y; a.mean = mean; a.rstd = rstd;
  a.pre_c = (const bf16*)pre_c; a.pre_nc = (const bf16*)pre_nc;
  a.N = N; a.HW = HW; a.C = C; a.G = G; a.silu = silu; a.eps = eps;
  return run<false>(a, ws, (cudaStream_t)stream);
}

// dx, the parameter gradients dw / db [C] and those of pre_c / pre_nc (bf16; null: not wanted). accumulate: bit 0 adds
// into dw, bit 1 into db, bit 2 into dpre_c.
int eri_gn_bwd(const void* x, const void* pre_c, const void* pre_nc, const void* dy, const void* w, const void* b,
               const float* mean, const float* rstd, void* dx, void* dw, void* db, void* dpre_c, void* dpre_nc, float* ws,
               int N, int HW, int C, int G, int silu, int accumulate, void* stream) {
  if (N < 1 || HW < 1 || C < 8 || G < 1 || C % 8 || C % G) return -1;
  GnArgs a = {};
  a.x = (const bf16*)x; a.dy = (const bf16*)dy; a.w = (const bf16*)w; a.b = (const bf16*)b;
  a.pre_c = (const bf16*)pre_c; a.pre_nc = (const bf16*)pre_nc;
  a.mean = const_cast<float*>(mean); a.rstd = const_cast<float*>(rstd);
  a.out = (bf16*)dx; a.dw = (bf16*)dw; a.db = (bf16*)db; a.dpre_c = (bf16*)dpre_c; a.dpre_nc = (bf16*)dpre_nc;
  a.N = N; a.HW = HW; a.C = C; a.G = G; a.silu = silu; a.accumulate = accumulate;
  return run<true>(a, ws, (cudaStream_t)stream);
}

}  // extern "C"
