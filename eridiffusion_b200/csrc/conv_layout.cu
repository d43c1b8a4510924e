// Convolution weights between the parameter order [Co, Ci, T] (T = kernel height x width) and the channels-last order
// [Co, T, Ci] that the convolutions read and their weight gradients come in.
//
// What bounds it: DRAM traffic (29 MB per order for a 1280 x 1280 x 3 x 3 weight). A CTA moves 256 input channels of one
// output channel through shared memory, so that both sides are read and written in 16-byte words; the gradient's
// transposition and its sum into the parameter's gradient are one pass. The copy is made in every forward pass and kept for
// that pass's backward, which reads it too: between the two, a network's convolution weights are held twice (1 GB more
// for a UNet of the SDXL widths); making it again in the backward would cost another 9 us per such weight.
// The library's strided copy took 18.6 us per such weight in each direction and its strided add 18.9 us, against 8.9 and
// 13.3 us of traffic.
#include "ptx.cuh"

using namespace eri;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int kC = 256, kMaxT = 25;

// ADD false: dst [Co, T, Ci] = src [Co, Ci, T]. ADD true: dst [Co, Ci, T] += src [Co, T, Ci]. Ci is a multiple of 8.
template <bool ADD>
__global__ void __launch_bounds__(256) weight_order_kernel(const bf16* __restrict__ src, bf16* __restrict__ dst, int Ci, int T) {
  extern __shared__ __align__(16) bf16 tile[];       // [channel][T]
  const int co = blockIdx.y, c0 = blockIdx.x * kC, n = min(kC, Ci - c0);
  const size_t flat = ((size_t)co * Ci + c0) * T;      // this CTA's run in the parameter order
  const int nv = n * T / 8, cv = n / 8;
  if (!ADD) {
    for (int i = threadIdx.x; i < nv; i += blockDim.x)
      reinterpret_cast<bf16x8*>(tile)[i] = reinterpret_cast<const bf16x8*>(src + flat)[i];
    __syncthreads();
    for (int i = threadIdx.x; i < cv * T; i += blockDim.x) {
      const int t = i / cv, c = (i - t * cv) * 8;
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(tile[(c + j) * T + t]);
      *reinterpret_cast<bf16x8*>(dst + ((size_t)co * T + t) * Ci + c0 + c) = pack8(f);
    }
  } else {
    for (int i = threadIdx.x; i < cv * T; i += blockDim.x) {
      const int t = i / cv, c = (i - t * cv) * 8;
      float f[8];
      unpack8(*reinterpret_cast<const bf16x8*>(src + ((size_t)co * T + t) * Ci + c0 + c), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) tile[(c + j) * T + t] = __float2bfloat16(f[j]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
      bf16x8* o = reinterpret_cast<bf16x8*>(dst + flat) + i;
      float a[8], b[8];
      unpack8(*o, a);
      unpack8(reinterpret_cast<const bf16x8*>(tile)[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
      *o = pack8(a);
    }
  }
}

}  // namespace

extern "C" int eri_conv_weight_order(const void* src, void* dst, int Co, int Ci, int T, int add, void* stream) {
  if (Co < 1 || Co > 65535 || Ci % 8 || Ci < 8 || T < 1 || T > kMaxT) return -1;
  if (((uintptr_t)src | (uintptr_t)dst) & 15) return -1;
  const dim3 grid((Ci + kC - 1) / kC, Co);
  const int smem = kC * T * (int)sizeof(bf16);
  if (add)
    weight_order_kernel<true><<<grid, 256, smem, (cudaStream_t)stream>>>((const bf16*)src, (bf16*)dst, Ci, T);
  else
    weight_order_kernel<false><<<grid, 256, smem, (cudaStream_t)stream>>>((const bf16*)src, (bf16*)dst, Ci, T);
  return (int)cudaGetLastError();
}
