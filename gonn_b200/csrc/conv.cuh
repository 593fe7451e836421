// Shared by the convolution kernels (conv.cu, conv_cl.cu).
#pragma once
#include "common.cuh"

namespace gbc {

__device__ __forceinline__ float raw16_to_float(uint16_t u, int bf) {
  return bf ? __uint_as_float((uint32_t)u << 16) : __half2float(__ushort_as_half(u));
}
__device__ __forceinline__ uint16_t float_to_raw16(float v, int bf) {
  return bf ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

// dW (M, C, T) (+)= sum over splits of part [splits][M][K] (conv.cu); tap_major: columns of part are (tap, c), else (c, tap).
int launch_wgrad_finish(const float* part, uint16_t* dW, int M, int C, int T, int splits, int bf16, int beta, bool tap_major,
                        cudaStream_t s);

}  // namespace gbc
