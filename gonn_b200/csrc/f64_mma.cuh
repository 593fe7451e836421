// The double-precision tensor instruction of the fp64 products (gemm_exact.cu) and the fp64 attention (attn_f64.cu).
#pragma once
#include "common.cuh"

namespace gb {

// A (16 x 8): a0 (g, t), a1 (g + 8, t), a2 (g, t + 4), a3 (g + 8, t + 4); B (8 x 8): b0 (t, g), b1 (t + 4, g);
// C (16 x 8): c0, c1 (g, 2t + {0, 1}), c2, c3 (g + 8, 2t + {0, 1}); g = lane / 4, t = lane % 4.
__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double a2, double a3, double b0, double b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

}  // namespace gb
