// RMS norm over the whole channel width followed by rotary embedding of interleaved pairs, for the query and key
// columns of a packed projection [rows, 3 * D], forward and backward (the LTX-style video blocks: one norm and one
// table row per token, not per head).
//
// What bounds it: DRAM traffic. At 19008 tokens x 4096 the two table rows of a token (16 KB fp32) are as large as q
// and k together, so one CTA takes both halves of a token and reads the tables once: forward 0.93 GB, backward
// 1.25 GB. A CTA holds a whole token in registers (the sums need a block reduction, nothing is read twice), and
// q, k are read inside the projection's output and their gradients written inside its gradient.
// As separate fp32 passes (contiguous copies, norm, two multiplies, add, stack, cast per operand and direction) the
// same work took 7.2 ms of a 47 ms training pass over one block at 19008 tokens; the pass with this kernel takes 41-42 ms.
// Reference: src/models/ltx2_model.rs:180-260 (QK-norm across heads, rotary over the inner dimension).
#include "ptx.cuh"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

struct NormRopeArgs {
  const bf16 *x[2], *w[2];   // q and k columns (row stride ldx), their norm weights [D]
  const float *cos, *sin;    // [L, D / 2], row stride ldt
  bf16* y[2];                // forward: [rows, D]
  const bf16* dy[2];         // backward: [rows, D]
  bf16* dx[2];               // backward: columns of the projection's gradient (row stride lddx)
  float* rstd;               // [2, rows]
  long long ldx, lddx, ldt;
  int rows, L, D;
  float eps;
};

constexpr int kThreads = 256;

// Sums of a and b over the block; `sm` is used once per kernel.
__device__ __forceinline__ float2 block_sum2(float a, float b, float2* sm) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = make_float2(a, b);
  __syncthreads();
  float2 t = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) {
    t.x += sm[i].x;
    t.y += sm[i].y;
  }
  return t;
}

__device__ __forceinline__ void load_table(const NormRopeArgs& a, int row, int vec, float4& c, float4& s) {
  const size_t o = (size_t)(row % a.L) * a.ldt + vec * 4;
  c = __ldg(reinterpret_cast<const float4*>(a.cos + o));
  s = __ldg(reinterpret_cast<const float4*>(a.sin + o));
}
// f rotated by +angle (dir = 1) or -angle (dir = -1: the gradient).
__device__ __forceinline__ void rotate8(float (&f)[8], const float4& c, const float4& s, float dir) {
  const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {s.x * dir, s.y * dir, s.z * dir, s.w * dir};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x0 = f[2 * i], x1 = f[2 * i + 1];
    f[2 * i] = cc[i] * x0 - ss[i] * x1;
    f[2 * i + 1] = ss[i] * x0 + cc[i] * x1;
  }
}

// V: 16-byte vectors per thread and operand (D <= 8 * V * kThreads).
template <int V>
__global__ void __launch_bounds__(kThreads) norm_rope_fwd_kernel(const NormRopeArgs a) {
  __shared__ float2 sm[kThreads / 32];
  const int row = blockIdx.x, nvec = a.D >> 3;
  bf16x8 q[2][V];
  float ss[2] = {0.f, 0.f};
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int v = threadIdx.x + u * kThreads;
    if (v < nvec)
#pragma unroll
      for (int o = 0; o < 2; ++o) q[o][u] = reinterpret_cast<const bf16x8*>(a.x[o] + (size_t)row * a.ldx)[v];
  }
#pragma unroll
  for (int u = 0; u < V; ++u)
    if (threadIdx.x + u * kThreads < nvec)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        float f[8];
        unpack8(q[o][u], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss[o] = fmaf(f[j], f[j], ss[o]);
      }
  const float2 t = block_sum2(ss[0], ss[1], sm);
  const float inv_d = 1.f / (float)a.D;
  const float rs[2] = {rsqrtf(t.x * inv_d + a.eps), rsqrtf(t.y * inv_d + a.eps)};
  if (threadIdx.x < 2 && a.rstd) a.rstd[(size_t)threadIdx.x * a.rows + row] = threadIdx.x ? rs[1] : rs[0];
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int v = threadIdx.x + u * kThreads;
    if (v >= nvec) continue;
    float4 c, s;
    load_table(a, row, v, c, s);
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      float f[8], w[8];
      unpack8(q[o][u], f);
      unpack8(reinterpret_cast<const bf16x8*>(a.w[o])[v], w);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] *= rs[o] * w[j];
      rotate8(f, c, s, 1.f);
      reinterpret_cast<bf16x8*>(a.y[o] + (size_t)row * a.D)[v] = pack8(f);
    }
  }
}

// g = rotate(dy, -angle) * w;  dx = rstd * (g - xhat * mean(g * xhat))
template <int V>
__global__ void __launch_bounds__(kThreads) norm_rope_bwd_kernel(const NormRopeArgs a) {
  __shared__ float2 sm[kThreads / 32];
  const int row = blockIdx.x, nvec = a.D >> 3;
  const float rs[2] = {a.rstd[row], a.rstd[(size_t)a.rows + row]};
  bf16x8 q[2][V], d[2][V];
  float4 c[V], s[V];
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int v = threadIdx.x + u * kThreads;
    if (v < nvec) {
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        q[o][u] = reinterpret_cast<const bf16x8*>(a.x[o] + (size_t)row * a.ldx)[v];
        d[o][u] = reinterpret_cast<const bf16x8*>(a.dy[o] + (size_t)row * a.D)[v];
      }
      load_table(a, row, v, c[u], s[u]);
    }
  }
  float dot[2] = {0.f, 0.f};
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int v = threadIdx.x + u * kThreads;
    if (v < nvec)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        float f[8], g[8], w[8];
        unpack8(q[o][u], f);
        unpack8(d[o][u], g);
        unpack8(reinterpret_cast<const bf16x8*>(a.w[o])[v], w);
        rotate8(g, c[u], s[u], -1.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) dot[o] = fmaf(g[j] * w[j], f[j] * rs[o], dot[o]);
      }
  }
  const float2 t = block_sum2(dot[0], dot[1], sm);
  const float inv_d = 1.f / (float)a.D, mean[2] = {t.x * inv_d, t.y * inv_d};
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int v = threadIdx.x + u * kThreads;
    if (v < nvec)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        float f[8], g[8], w[8];
        unpack8(q[o][u], f);
        unpack8(d[o][u], g);
        unpack8(reinterpret_cast<const bf16x8*>(a.w[o])[v], w);
        rotate8(g, c[u], s[u], -1.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = rs[o] * (g[j] * w[j] - f[j] * rs[o] * mean[o]);
        reinterpret_cast<bf16x8*>(a.dx[o] + (size_t)row * a.lddx)[v] = pack8(g);
      }
  }
}

}  // namespace

extern "C" {

// q, k: two [rows, D] operands of row stride ldx; yq, yk [rows, D] contiguous; rstd [2, rows] or null. Every pointer
// is 16-byte aligned, D and the strides are multiples of 8 (the tables' of 4); D <= 8192.
int eri_norm_rope_fwd(const void* q, const void* k, long long ldx, const void* wq, const void* wk, const float* cos,
                      const float* sin, long long ldt, void* yq, void* yk, float* rstd, int rows, int L, int D, float eps,
                      void* stream) {
  if (D % 8 || ldx % 8 || ldt % 4 || D > 8192 || L < 1) return -1;
  if (rows == 0) return 0;
  NormRopeArgs a = {};
  a.x[0] = (const bf16*)q; a.x[1] = (const bf16*)k; a.w[0] = (const bf16*)wq; a.w[1] = (const bf16*)wk;
  a.cos = cos; a.sin = sin; a.y[0] = (bf16*)yq; a.y[1] = (bf16*)yk; a.rstd = rstd;
  a.ldx = ldx; a.ldt = ldt; a.rows = rows; a.L = L; a.D = D; a.eps = eps;
  cudaStream_t st = (cudaStream_t)stream;
  if (D <= 2048) norm_rope_fwd_kernel<1><<<rows, kThreads, 0, st>>>(a);
  else if (D <= 4096) norm_rope_fwd_kernel<2><<<rows, kThreads, 0, st>>>(a);
  else norm_rope_fwd_kernel<4><<<rows, kThreads, 0, st>>>(a);
  return (int)cudaGetLastError();
}

// dyq, dyk [rows, D] contiguous; dq, dk: [rows, D] of row stride lddx.
int eri_norm_rope_bwd(const void* q, const void* k, long long ldx, const void* wq, const void* wk, const float* cos,
                      const float* sin, long long ldt, const float* rstd, const void* dyq, const void* dyk, void* dq,
                      void* dk, long long lddx, int rows, int L, int D, void* stream) {
  if (D % 8 || ldx % 8 || lddx % 8 || ldt % 4 || D > 8192 || L < 1) return -1;
  if (rows == 0) return 0;
  NormRopeArgs a = {};
  a.x[0] = (const bf16*)q; a.x[1] = (const bf16*)k; a.w[0] = (const bf16*)wq; a.w[1] = (const bf16*)wk;
  a.cos = cos; a.sin = sin; a.dy[0] = (const bf16*)dyq; a.dy[1] = (const bf16*)dyk; a.dx[0] = (bf16*)dq; a.dx[1] = (bf16*)dk;
  a.rstd = const_cast<float*>(rstd);
  a.ldx = ldx; a.lddx = lddx; a.ldt = ldt; a.rows = rows; a.L = L; a.D = D;
  cudaStream_t st = (cudaStream_t)stream;
  if (D <= 2048) norm_rope_bwd_kernel<1><<<rows, kThreads, 0, st>>>(a);
  else if (D <= 4096) norm_rope_bwd_kernel<2><<<rows, kThreads, 0, st>>>(a);
  else norm_rope_bwd_kernel<4><<<rows, kThreads, 0, st>>>(a);
  return (int)cudaGetLastError();
}

}  // extern "C"
