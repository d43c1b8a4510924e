// Column reductions over the rows of [rows, N] bf16 matrices: the gradients of biases, norm parameters and adaLN
// modulation. One launch each, results in bf16, optionally added into the parameter's gradient buffer.
//
//   sum    out[n]    = sum_r x[r, n]                                     bias gradient
//   norm   s0[b, n]  = sum_r dy[r, n],  s1[b, n] = sum_r dy[r, n] xhat[r, n]     (shift / bias, scale / weight)
//   dot    out[b, n] = sum_r x[r, n] y[r, n]                             gate gradient
//
// Bound by reading the operands once. A cluster of eight CTAs owns 64 columns of one batch element: eight lanes of
// 16 bytes cover a row's 128-byte segment, 32 row lanes walk the CTA's eighth of the rows with four loads in
// flight each, and the eight partial rows are added over distributed shared memory in CTA order (deterministic,
// no workspace). What they replace at [4096, 3072]: 13 us library reduction + 2 us add (sum), 62 us atomic kernel
// + fills and conversions (norm), 44 us (dot).
#include "ptx.cuh"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int kCols = 64, kRowLanes = 32, kSplit = 8;
enum Mode { kSum = 0, kNorm = 1, kDot = 2 };

struct ColArgs {
  const bf16 *x, *y;            // sum: x; norm: x = dy, y = the norm's input; dot: both factors
  const float *mean, *rstd;     // norm: per row (mean null: RMS norm)
  bf16 *out0, *out1;            // norm: s0, s1 (either may be null)
  long long ld;                 // row stride of x (and y)
  int rows, N, accumulate;      // rows per batch element; accumulate: bit 0 out0, bit 1 out1
};

template <int MODE>
__global__ void __cluster_dims__(1, kSplit, 1) __launch_bounds__(256) col_kernel(const ColArgs a) {
  constexpr int S = MODE == kNorm ? 2 : 1;
  constexpr int kInFlight = MODE == kSum ? 4 : 2;
  __shared__ float red[S][kRowLanes][kCols + 1];
  __shared__ float part[S][kCols];
  const int lane = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int col = blockIdx.x * kCols + lane * 8;
  const int per = (a.rows + kSplit - 1) / kSplit;
  const int r0 = blockIdx.y * per, r1 = min(a.rows, r0 + per);
  const size_t row_base = (size_t)blockIdx.z * a.rows;
  float s[S][8];
#pragma unroll
  for (int k = 0; k < S; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) s[k][j] = 0.f;
  if (col < a.N) {
    const bf16* px = a.x + row_base * a.ld + col;
    const bf16* py = MODE == kSum ? nullptr : a.y + row_base * a.ld + col;
    for (int r = r0 + rl; r < r1; r += kRowLanes * kInFlight) {
      bf16x8 q[kInFlight], t[kInFlight];
      float mu[kInFlight], rs[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const int rr = r + u * kRowLanes;
        if (rr < r1) {
          q[u] = *reinterpret_cast<const bf16x8*>(px + (size_t)rr * a.ld);
          if (MODE != kSum) t[u] = *reinterpret_cast<const bf16x8*>(py + (size_t)rr * a.ld);
          if (MODE == kNorm) {
            mu[u] = a.mean ? a.mean[row_base + rr] : 0.f;
            rs[u] = a.rstd[row_base + rr];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kInFlight; ++u)
        if (r + u * kRowLanes < r1) {
          float f[8], g[8];
          unpack8(q[u], f);
          if (MODE != kSum) unpack8(t[u], g);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (MODE == kDot) {
              s[0][j] = fmaf(f[j], g[j], s[0][j]);
            } else {
              s[0][j] += f[j];
              if constexpr (MODE == kNorm) s[1][j] = fmaf(f[j], (g[j] - mu[u]) * rs[u], s[1][j]);
            }
          }
        }
    }
  }
#pragma unroll
  for (int k = 0; k < S; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) red[k][rl][lane * 8 + j] = s[k][j];
  __syncthreads();
  // 256 threads: four per column, each over eight row lanes
  const int c = threadIdx.x >> 2, q4 = threadIdx.x & 3;
#pragma unroll
  for (int k = 0; k < S; ++k) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kRowLanes / 4; ++i) t += red[k][q4 * (kRowLanes / 4) + i][c];
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    if (q4 == 0) part[k][c] = t;
  }
  cluster_sync_all();
  if (blockIdx.y == 0 && threadIdx.x < S * kCols) {
    const int k = threadIdx.x / kCols, cc = threadIdx.x % kCols, oc = blockIdx.x * kCols + cc;
    bf16* out = k ? a.out1 : a.out0;
    if (out && oc < a.N) {
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < kSplit; ++i) v += ld_shared_cluster_f32(map_to_cta(smem_u32(&part[k][cc]), (uint32_t)i));
      out += (size_t)blockIdx.z * a.N + oc;
      if (a.accumulate & (1 << k)) v += __bfloat162float(*out);
      *out = __float2bfloat16(v);
    }
  }
  cluster_sync_all();      // the partial rows are read before their CTAs leave
}

template <int MODE>
int run(const ColArgs& a, int batches, cudaStream_t st) {
  if (a.rows < 1 || batches < 1 || batches > 65535 || a.N < 8 || a.N % 8 || a.ld % 8) return -1;
  if (((uintptr_t)a.x | (uintptr_t)a.y) & 15) return -1;
  col_kernel<MODE><<<dim3((a.N + kCols - 1) / kCols, kSplit, batches), 256, 0, st>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

// x [M, N] (row stride ld); N and ld multiples of 8, x 16-byte aligned; out [N].
int eri_col_sum(const void* x, long long ld, void* out, int M, int N, int accumulate, void* stream) {
  ColArgs a = {};
  a.x = (const bf16*)x; a.out0 = (bf16*)out; a.ld = ld; a.rows = M; a.N = N; a.accumulate = accumulate ? 1 : 0;
  return run<kSum>(a, 1, (cudaStream_t)stream);
}

// dy, x [batches * rows, D] contiguous; sum_dy / sum_dyx [batches, D] (null: not wanted). mean null: RMS norm.
int eri_col_norm_grad(const void* dy, const void* x, const float* mean, const float* rstd, void* sum_dy, void* sum_dyx,
                      int batches, int rows, int D, int accumulate, void* stream) {
  ColArgs a = {};
  a.x = (const bf16*)dy; a.y = (const bf16*)x; a.mean = mean; a.rstd = rstd; a.out0 = (bf16*)sum_dy; a.out1 = (bf16*)sum_dyx;
  a.ld = D; a.rows = rows; a.N = D; a.accumulate = accumulate;
  return run<kNorm>(a, batches, (cudaStream_t)stream);
}

// out [batches, D] = column sums of x * y, both [batches * rows, D] contiguous.
int eri_col_dot(const void* x, const void* y, void* out, int batches, int rows, int D, void* stream) {
  ColArgs a = {};
  a.x = (const bf16*)x; a.y = (const bf16*)y; a.out0 = (bf16*)out; a.ld = D; a.rows = rows; a.N = D;
  return run<kDot>(a, batches, (cudaStream_t)stream);
}

}  // extern "C"
