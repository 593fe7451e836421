// int8 quantisation support kernels: min / max reduction, affine q-parameters computed
// on the device (so dynamic quantisation needs no host round trip), quantise to int8
// with round-half-away-from-zero and clamping to [-128, 127], and fake quantisation
// with a clamped straight-through backward.
//
// Rules follow the reference (quant/quant.go:100-143): q = clamp(round(x / s) + zp);
// affine range nudged to include 0, scale = (max - min) / 255, zp = -128 - round(min / s)
// clamped, degenerate range -> (1, 0); symmetric scale = max|x| / 127.
#include "common.cuh"

using namespace gb;

namespace {

constexpr int kObserveThreads = 512;
constexpr int kObserveBlocks = 148 * 4;

// Running least and largest value of whole vectors.  16-bit types compare in pairs, as they are: a third of the instructions
// of a conversion and two fp32 comparisons per element.
template <typename T>
struct MinMax {
  float mn = INFINITY, mx = -INFINITY;
  __device__ __forceinline__ void add(const uint4& u) {
    const float v[4] = {__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w)};
#pragma unroll
    for (int k = 0; k < 4; k++) { mn = fminf(mn, v[k]); mx = fmaxf(mx, v[k]); }
  }
  __device__ __forceinline__ float least() const { return mn; }
  __device__ __forceinline__ float largest() const { return mx; }
};
template <typename T, typename T2>
struct MinMax2 {
  T2 mn, mx;
  __device__ __forceinline__ MinMax2(float inf) { mn.x = mn.y = (T)inf; mx.x = mx.y = (T)-inf; }
  __device__ __forceinline__ void add(const uint4& u) {
    const T2* e = reinterpret_cast<const T2*>(&u);
#pragma unroll
    for (int k = 0; k < 4; k++) { mn = __hmin2(mn, e[k]); mx = __hmax2(mx, e[k]); }
  }
  __device__ __forceinline__ float least() const { return fminf((float)mn.x, (float)mn.y); }
  __device__ __forceinline__ float largest() const { return fmaxf((float)mx.x, (float)mx.y); }
};
template <>
struct MinMax<__nv_bfloat16> : MinMax2<__nv_bfloat16, __nv_bfloat162> {
  __device__ __forceinline__ MinMax() : MinMax2(INFINITY) {}
};
template <>
struct MinMax<__half> : MinMax2<__half, __half2> {
  __device__ __forceinline__ MinMax() : MinMax2(INFINITY) {}
};

// Least and largest value of x, one pair per block (NaNs are passed over).  Bound by memory: four 16-byte loads in flight per
// thread; an x that is not 16-byte aligned, and the elements behind the last whole vector, go one by one.
// 8192 x 4096 bf16 (67 MB, behind a product whose result the L2 still has to write back): 16 us; 27 us with one 2-byte load
// at a time.
template <typename T>
__global__ void __launch_bounds__(kObserveThreads, 4) minmax_partial_kernel(const T* __restrict__ x, long long n, float* __restrict__ part) {
  __shared__ float red[32];
  constexpr int VEC = 16 / (int)sizeof(T);
  MinMax<T> acc;
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long nv = ((uintptr_t)x & 15) == 0 ? n / VEC : 0;
  const uint4* xv = reinterpret_cast<const uint4*>(x);
  long long i = first;
  for (; i < nv; i += 4 * stride) {
    uint4 u[4];
#pragma unroll
    for (int k = 0; k < 4; k++) u[k] = xv[min(i + k * stride, nv - 1)];   // (behind the end: the last vector again)
#pragma unroll
    for (int k = 0; k < 4; k++) acc.add(u[k]);
  }
  float mn = acc.least(), mx = acc.largest();
  for (i = nv * VEC + first; i < n; i += stride) {
    const float v = (float)x[i];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  mx = block_max(mx, red);
  mn = -block_max(-mn, red);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = mn;
    part[2 * blockIdx.x + 1] = mx;
  }
}

// The block's copy of the q-parameters of what minmax_partial_kernel left in `part`: {min, max, scale, zero point}.
__device__ __forceinline__ void qparams_of(const float* __restrict__ part, int nparts, int symmetric, float* out4) {
  __shared__ float red[32];
  float mn = INFINITY, mx = -INFINITY;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
    mn = fminf(mn, part[2 * i]);
    mx = fmaxf(mx, part[2 * i + 1]);
  }
  mx = block_max(mx, red);
  mn = -block_max(-mn, red);
  float scale;
  int zp = 0;
  if (symmetric) {
    float m = fmaxf(fabsf(mn), fabsf(mx));
    scale = m == 0.f ? 1.f : m / 127.f;
  } else {
    float lo = fminf(0.f, mn), hi = fmaxf(0.f, mx);
    scale = (hi - lo) / 255.f;
    if (scale == 0.f) {
      scale = 1.f;
      zp = 0;
    } else {
      zp = -128 - (int)roundf(lo / scale);
      zp = zp < -128 ? -128 : (zp > 127 ? 127 : zp);
    }
  }
  out4[0] = mn; out4[1] = mx; out4[2] = scale; out4[3] = (float)zp;
}

// out4: {min, max, scale, zero_point (as float)}; zp_int also written to zp_out
__global__ void qparams_kernel(const float* __restrict__ part, int nparts, int symmetric,
                               float* __restrict__ out4, int* __restrict__ zp_out) {
  float qp[4];
  qparams_of(part, nparts, symmetric, qp);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 4; k++) out4[k] = qp[k];
    if (zp_out) *zp_out = (int)qp[3];
  }
}

// round(x / s), halves away from zero: the sum with half of the sign is rounded towards zero, so that it reaches the next whole
// number only when x / s is at least half way to it.
template <typename T>
__device__ __forceinline__ int round_div(T x, float s) {
  const float t = (float)x / s;
  return __float2int_rz(__fadd_rz(t, copysignf(0.5f, t)));
}
// Two values clamped to a byte each in the lower half of a word, the lower half of `next` in its upper half.
__device__ __forceinline__ uint32_t pack_s8(int a, int b, uint32_t next) {
  uint32_t d;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(b), "r"(a), "r"(next));
  return d;
}
template <typename T>
__device__ __forceinline__ uint32_t quantize_four(const T* x, float s, int z) {
  return pack_s8(round_div(x[0], s) + z, round_div(x[1], s) + z, pack_s8(round_div(x[2], s) + z, round_div(x[3], s) + z, 0u));
}
template <typename T>
__device__ __forceinline__ int8_t quantize_one(T x, float s, int z) {
  const int v = round_div(x, s) + z;
  return (int8_t)(v < -128 ? -128 : (v > 127 ? 127 : v));
}
template <typename T>
__device__ __forceinline__ uint4 quantize_sixteen(const T* x, float s, int z) {
  return make_uint4(quantize_four(x, s, z), quantize_four(x + 4, s, z), quantize_four(x + 8, s, z), quantize_four(x + 12, s, z));
}

template <typename T>
__global__ void quantize_kernel(const T* __restrict__ x, int8_t* __restrict__ q, long long rows,
                                long long cols, long long ldq, const float* __restrict__ scale,
                                const int* __restrict__ zp, int per_row) {
  const long long n = rows * cols;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / cols, c = i - r * cols;
    const float s = per_row ? scale[r] : scale[0];
    const int z = zp ? (per_row ? zp[r] : zp[0]) : 0;
    q[r * ldq + c] = quantize_one(x[i], s, z);
  }
}

// Sixteen elements per thread: 16-byte stores of the int8 output, 16-byte loads of the input.
// Needs cols and ldq to be multiples of 16 and both base pointers 16-byte aligned, so that a
// group of sixteen never straddles a row.
template <typename T>
__global__ void quantize_vec_kernel(const T* __restrict__ x, int8_t* __restrict__ q, long long rows,
                                    long long cols, long long ldq, const float* __restrict__ scale,
                                    const int* __restrict__ zp, int per_row) {
  const long long groups = rows * cols / 16;
  const long long gpr = cols / 16;
  constexpr int LD = 16 / (int)sizeof(T);          // elements per 16-byte load
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < groups;
       g += (long long)gridDim.x * blockDim.x) {
    const long long r = g / gpr, c = (g - r * gpr) * 16;
    const float s = per_row ? scale[r] : scale[0];
    const int z = zp ? (per_row ? zp[r] : zp[0]) : 0;
    alignas(16) T v[16];
#pragma unroll
    for (int k = 0; k < 16 / LD; ++k)
      *reinterpret_cast<uint4*>(&v[k * LD]) = *reinterpret_cast<const uint4*>(x + r * cols + c + k * LD);
    *reinterpret_cast<uint4*>(q + r * ldq + c) = quantize_sixteen(v, s, z);
  }
}

// Dynamic quantisation behind minmax_partial_kernel: every block works the q-parameters out of the partial results for itself
// (592 pairs from L2, about 2 us, instead of a launch of one block between the two) and block 0 writes them for the product.
// Whole rows of 16-byte vectors are one flat array (VEC: cols == ldq, 16-byte aligned, a multiple of 16 elements), walked
// from its end, since the last vectors that the observing pass read are still in L2.  8192 x 4096 bf16: 16 us, with the
// launch between them 22 us before.
template <typename T, bool VEC>
__global__ void __launch_bounds__(kObserveThreads, 4) quantize_dynamic_kernel(const T* __restrict__ x, int8_t* __restrict__ q, long long rows, long long cols,
                                                                           long long ldq, const float* __restrict__ part, int nparts,
                                                                           float* __restrict__ out4, int* __restrict__ zp_out) {
  float qp[4];
  qparams_of(part, nparts, 0, qp);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (int k = 0; k < 4; k++) out4[k] = qp[k];
    *zp_out = (int)qp[3];
  }
  const float s = qp[2];
  const int z = (int)qp[3];
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  if (VEC) {
    constexpr int LD = 16 / (int)sizeof(T);
    const long long groups = rows * cols / 16;
    for (long long g = groups - 1 - first; g >= 0; g -= stride) {
      uint4 u[16 / LD];
#pragma unroll
      for (int k = 0; k < 16 / LD; ++k) u[k] = reinterpret_cast<const uint4*>(x)[g * (16 / LD) + k];
      reinterpret_cast<uint4*>(q)[g] = quantize_sixteen(reinterpret_cast<const T*>(u), s, z);
    }
  } else {
    // the padding of a row (columns cols .. ldq - 1) becomes zero here
    for (long long i = first; i < rows * ldq; i += stride) {
      const long long r = i / ldq, c = i - r * ldq;
      q[i] = c < cols ? quantize_one(x[r * cols + c], s, z) : (int8_t)0;
    }
  }
}

// MODE 0: y = (q(x) - zp) * s;  MODE 1: dx = dy where x lies inside the representable range
template <typename T, int MODE>
__global__ void fake_quant_kernel(const T* __restrict__ x, const T* __restrict__ dy, T* __restrict__ y,
                                  long long n, const float* __restrict__ qp) {
  const float s = qp[0];
  const int zp = (int)qp[1];
  const float lo = (-128.f - zp) * s, hi = (127.f - zp) * s;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = (float)x[i];
    if (MODE == 0) {
      int q = (int)roundf(v / s) + zp;
      q = q < -128 ? -128 : (q > 127 ? 127 : q);
      y[i] = (T)((float)(q - zp) * s);
    } else {
      y[i] = (v >= lo && v <= hi) ? dy[i] : (T)0.f;
    }
  }
}

inline int grid_for(long long n) {
  long long g = (n + 255) / 256;
  if (g > 148 * 8) g = 148 * 8;
  return g < 1 ? 1 : (int)g;
}

// Blocks of the observing pass: a thread has sixteen elements or more until every SM has its four blocks.
inline int observe_grid(long long n) {
  const long long g = (n + kObserveThreads * 16 - 1) / (kObserveThreads * 16);
  return g < 1 ? 1 : g > kObserveBlocks ? kObserveBlocks : (int)g;
}

}  // namespace

enum { DT_BF16 = 0, DT_F16 = 1, DT_F32 = 2 };

#define GB_Q_DISPATCH(CALL)                                   \
  switch (dtype) {                                            \
    case DT_BF16: { using T = __nv_bfloat16; CALL; } break;   \
    case DT_F16: { using T = __half; CALL; } break;           \
    case DT_F32: { using T = float; CALL; } break;            \
    default:                                                  \
      gbh::set_error("quant: unsupported dtype %d", dtype);   \
      return gbh::E_BAD_ARG;                                  \
  }

GB_EXPORT int gb_q_scratch_floats() { return 2 * kObserveBlocks; }

// Observes x: out4 = {min, max, scale, zero_point}; zp_out (int, may be null) gets the
// zero point.  scratch: gb_q_scratch_floats() floats.
GB_EXPORT int gb_q_observe(int dtype, const void* x, long long n, int symmetric, float* scratch,
                           float* out4, int* zp_out, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const int g = observe_grid(n);
  GB_Q_DISPATCH((minmax_partial_kernel<T><<<g, kObserveThreads, 0, s>>>((const T*)x, n, scratch)));
  qparams_kernel<<<1, 256, 0, s>>>(scratch, g, symmetric, out4, zp_out);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// Observes x (rows x cols, contiguous) and quantises it with the affine q-parameters that it finds, in two launches: out4 and
// zp_out as gb_q_observe leaves them, q as gb_q_quantize does, with zeros in the padding of its rows (ldq >= cols bytes apart).
// scratch: gb_q_scratch_floats() floats.
GB_EXPORT int gb_q_dynamic(int dtype, const void* x, void* q, long long rows, long long cols, long long ldq, float* scratch,
                           float* out4, int* zp_out, void* stream) {
  if (rows <= 0 || cols <= 0 || ldq < cols) {
    gbh::set_error("gb_q_dynamic: bad extents %lld x %lld, pitch %lld", rows, cols, ldq);
    return gbh::E_BAD_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const long long n = rows * cols;
  const int g = observe_grid(n);
  GB_Q_DISPATCH((minmax_partial_kernel<T><<<g, kObserveThreads, 0, s>>>((const T*)x, n, scratch)));
  const bool vec = cols == ldq && n % 16 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)q & 15) == 0;
  if (vec) {
    GB_Q_DISPATCH((quantize_dynamic_kernel<T, true><<<g, kObserveThreads, 0, s>>>((const T*)x, (int8_t*)q, rows, cols, ldq, scratch, g, out4, zp_out)));
  } else {
    GB_Q_DISPATCH((quantize_dynamic_kernel<T, false><<<g, kObserveThreads, 0, s>>>((const T*)x, (int8_t*)q, rows, cols, ldq, scratch, g, out4, zp_out)));
  }
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// q[r][c] = clamp(round(x[r][c] / scale) + zp); scale / zp are device scalars, or one
// value per row when per_row != 0; zp may be null (0).  ldq: row pitch of q in bytes.
GB_EXPORT int gb_q_quantize(int dtype, const void* x, void* q, long long rows, long long cols,
                            long long ldq, const float* scale, const int* zp, int per_row,
                            void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (rows * cols <= 0) return gbh::E_OK;
  const bool vec = cols % 16 == 0 && ldq % 16 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)q & 15) == 0;
  if (vec) {
    GB_Q_DISPATCH((quantize_vec_kernel<T><<<grid_for(rows * cols / 16), 256, 0, s>>>((const T*)x, (int8_t*)q, rows, cols, ldq, scale, zp, per_row)));
  } else {
    GB_Q_DISPATCH((quantize_kernel<T><<<grid_for(rows * cols), 256, 0, s>>>((const T*)x, (int8_t*)q, rows, cols, ldq, scale, zp, per_row)));
  }
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// mode 0: fake-quantise x into y; mode 1: straight-through gradient (x, dy -> y).
// qp: device pair {scale, zero_point as float}.
GB_EXPORT int gb_fake_quant(int mode, int dtype, const void* x, const void* dy, void* y, long long n,
                            const float* qp, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n <= 0) return gbh::E_OK;
  if (mode == 0) {
    GB_Q_DISPATCH((fake_quant_kernel<T, 0><<<grid_for(n), 256, 0, s>>>((const T*)x, nullptr, (T*)y, n, qp)));
  } else {
    GB_Q_DISPATCH((fake_quant_kernel<T, 1><<<grid_for(n), 256, 0, s>>>((const T*)x, (const T*)dy, (T*)y, n, qp)));
  }
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}
