// Token strides (elements between consecutive tokens) of the attention operands; 0 = contiguous [B, L, H, DH].
// Heads are packed (DH apart), batches L * stride apart, strides multiples of 8: a column block of a wider
// [B * L, stride] matrix, such as the q, k or v part of a projection's output.
#pragma once
extern "C" {
struct EriAttnStrides {
  long long q, k, v, out, dq, dk, dv;
};
}
