// Exact-precision GEMMs on tensor cores.
//
// The reference's float64 / float32 products are cuBLAS Dgemm / Sgemm calls
// (backend/cuda/gonn_cuda.cu:147-177, 255-294, 616-622).  tcgen05 has no fp64 or fp32 form, so:
//
// * fp64: mma.sync m16n8k8 f64 on 64 x 64 x 16 tiles.  Results match an fp64 FMA chain over k up to the order of
//   the sum (1e-13-class agreement with a float64 oracle).
// * fp32: each operand is split once into three bf16 planes (x = hi + mid + lo, 24 mantissa
//   bits in total) and the six significant plane products lo hi, hi lo, mid mid, mid hi, hi mid, hi hi
//   run as one bf16 tcgen05 launch, in that order into one fp32 accumulator; the planes are the third
//   dimension of the operands' tensor maps.  The dropped products are below 2^-24 of the result, the
//   rounding level of an fp32 product itself.  Infinities and NaN give what they give in fp32 (split3_kernel).
//   3000 x 4096 x 1024: 115 us (240 as three launches that added to C).
//
// The in-library benchmark loops at the end mirror the reference's (gonn_cuda.cu:255-294,
// 532-592, 673-690): operands allocated once, five untimed calls, `iters` calls between two
// events, milliseconds per call returned.
#include "f64_mma.cuh"

using namespace gb;

extern "C" int gb_gemm16(const void* A, const void* B, void* C, const void* bias, int bias_f32, void* aux, int M,
                         int N, int K, int batch, int transA, int transB, long long lda, long long ldb,
                         long long ldc, long long ldaux, long long sA, long long sB, long long sC, long long sAux,
                         int in_dtype, int out_dtype, int act, int aux_mode, int beta, float alpha, int force_bn,
                         void* workspace, long long workspace_bytes, void* stream);
int gemm_bf16_planes(const void* A, const void* B, float* C, const float* bias, int M, int N, int K, int batch, int transA,
                     int transB, long long lda, long long ldb, long long ldc, long long plane_a, long long plane_b, int bcastA,
                     int bcastB, long long sC, int planes, uint32_t order_a, uint32_t order_b, float alpha, int beta,
                     void* workspace, long long workspace_bytes, cudaStream_t stream, int chain, const unsigned* guard, int guard_top);
int gemm_fma_unless_planes(const void* A, const void* B, float* C, const float* bias, int M, int N, int K, int batch, int transA, int transB,
                           long long lda, long long ldb, long long ldc, long long sA, long long sB, long long sC, float alpha, int beta,
                           const unsigned* guard, int guard_top, cudaStream_t stream);
extern "C" int gb_binary(int op, int dtype, const void* a, const void* b, void* c, long long n, int rank,
                         const long long* shape, const long long* sa, const long long* sb, void* stream);
extern "C" int gb_flash_fwd(int dtype, const void* q, const void* k, const void* v, void* o, float* lse, int B, int H,
                            int Sq, int Sk, int D, long long q_sb, long long q_ss, long long q_sh, long long k_sb,
                            long long k_ss, long long k_sh, long long v_sb, long long v_ss, long long v_sh,
                            long long o_sb, long long o_ss, long long o_sh, float scale, int causal, void* stream);

namespace {

enum { DT_BF16 = 0, DT_F16 = 1, DT_F32 = 2, DT_F64 = 3 };

// ---------------------------------------------------------------------------
// fp64: mma.sync m16n8k8
// ---------------------------------------------------------------------------
// Bound by the fp64 tensor pipe (64 multiply-adds per SM and clock).  128 x 128 tiles of one 512-thread CTA kept
// it 68 % active: half the stalls were shared-memory instructions (8-byte fragments and 8-byte copies) and the
// barrier that all 16 warps share, and 256 such tiles leave 14 % of two waves empty at 2048^3 (790 us, now 558; 512^3 102, now 17).  Here a CTA
// is 64 x 64 x 16 with four warps of 32 x 32, four CTAs per SM that wait for nobody else's barrier, and
//  * an operand whose contiguous dimension is k is staged as [8-wide k block][row][8]: 16-byte copies, and one
//    16-byte read gives a lane the elements k = 2t and 2t + 1 of a row, which stand in the fragment's slots t and
//    t + 4 on both sides (the order of the contraction within a block of eight is free);
//  * the other form is staged as [k][row] with pitch 66: rows 2t and 2t + 1 are read without bank conflicts;
//  * when the tiles alone leave SMs idle, a cluster of 2, 4 or 8 CTAs cuts K and adds its parts through
//    distributed shared memory in rank order: no workspace, no second launch, deterministic.
constexpr int DB = 64, DBK = 16, DSTAGES = 3;
constexpr int DTHREADS = 128;
constexpr int DPITCH = DB + 2;                          // [k][row] form
constexpr int DOP = DBK * DPITCH;                       // doubles of one operand stage (the larger form)
constexpr int DSMEM = DSTAGES * 2 * DOP * 8;
static_assert(DB * DB <= DSTAGES * 2 * DOP, "the cluster's partial tiles reuse the stages");

// 64 rows (of MN) x 16 k of an operand into a stage.  KC: stored (MN, K), else (K, MN); k runs to k_end.
template <bool KC>
__device__ __forceinline__ void load_tile(double* st, const double* src, long long ld, int mn0, int k0, int MN, int k_end, bool vec) {
  if (vec) {
#pragma unroll
    for (int i = 0; i < DB * DBK / 2 / DTHREADS; i++) {
      const int q = threadIdx.x + i * DTHREADS;
      if (KC) {
        const int r = q >> 3, c = q & 7, k = k0 + 2 * c;
        const int have = mn0 + r < MN ? min(2, max(0, k_end - k)) * 8 : 0;
        cp_async16(st + ((c >> 2) * DB + r) * 8 + (c & 3) * 2, have ? src + (long long)(mn0 + r) * ld + k : src, have);
      } else {
        const int kk = q >> 5, c = (q & 31) * 2, k = k0 + kk;
        const int have = k < k_end ? min(2, max(0, MN - mn0 - c)) * 8 : 0;
        cp_async16(st + kk * DPITCH + c, have ? src + (long long)k * ld + mn0 + c : src, have);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < DB * DBK / DTHREADS; i++) {
      const int q = threadIdx.x + i * DTHREADS;
      const int r = KC ? q >> 4 : q & 63, kk = KC ? q & 15 : q >> 6;
      const bool ok = mn0 + r < MN && k0 + kk < k_end;
      const long long at = KC ? (long long)(mn0 + r) * ld + k0 + kk : (long long)(k0 + kk) * ld + mn0 + r;
      cp_async8(KC ? st + ((kk >> 3) * DB + r) * 8 + (kk & 7) : st + kk * DPITCH + r, ok ? src + at : src, ok ? 8 : 0);
    }
  }
}
// Elements k = 2t and 2t + 1 of k block kb, row r.
template <bool KC>
__device__ __forceinline__ void frag(const double* st, int kb, int t, int r, double& lo, double& hi) {
  if (KC) {
    const double2 v = *reinterpret_cast<const double2*>(st + (kb * DB + r) * 8 + 2 * t);
    lo = v.x; hi = v.y;
  } else {
    lo = st[(kb * 8 + 2 * t) * DPITCH + r];
    hi = st[(kb * 8 + 2 * t + 1) * DPITCH + r];
  }
}

// grid: (row tiles * column tiles * splits, batch); a cluster is the `splits` CTAs of one tile.
template <bool AK, bool BKC>
__global__ void __launch_bounds__(DTHREADS, 4)
gemm_f64_mma_kernel(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C, int M, int N, int K,
                    long long lda, long long ldb, long long ldc, long long sA, long long sB, long long sC, double alpha, int beta,
                    int splits, int k_per) {
  extern __shared__ __align__(16) double dsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const unsigned tile = splits == 1 ? blockIdx.x : blockIdx.x / splits, tiles_n = (N + DB - 1) / DB;
  const int rank = (int)(blockIdx.x - tile * splits);
  const int m0 = (int)(tile / tiles_n) * DB, n0 = (int)(tile % tiles_n) * DB;
  A += (long long)blockIdx.y * sA;
  B += (long long)blockIdx.y * sB;
  C += (long long)blockIdx.y * sC;
  const bool a_vec = ((lda & 1) == 0) && (((uintptr_t)A & 15) == 0);
  const bool b_vec = ((ldb & 1) == 0) && (((uintptr_t)B & 15) == 0);
  const int k_begin = rank * k_per, k_end = min(K, k_begin + k_per);
  const int nk = k_end > k_begin ? (k_end - k_begin + DBK - 1) / DBK : 0;
  double acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[i][j][e] = 0.0;

  auto issue = [&](int kt) {
    if (kt < nk) {
      double* st = dsm + (kt % DSTAGES) * 2 * DOP;
      load_tile<AK>(st, A, lda, m0, k_begin + kt * DBK, M, k_end, a_vec);
      load_tile<BKC>(st + DOP, B, ldb, n0, k_begin + kt * DBK, N, k_end, b_vec);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < DSTAGES - 1; i++) issue(i);
  for (int kt = 0; kt < nk; kt++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DSTAGES - 2) : "memory");   // tile kt has landed
    __syncthreads();                                                         // ... for every thread; kt - 1 is no longer read
    issue(kt + DSTAGES - 1);
    const double* sa = dsm + (kt % DSTAGES) * 2 * DOP;
    const double* sb = sa + DOP;
#pragma unroll
    for (int kb = 0; kb < DBK / 8; kb++) {
      double af[2][4], bf[4][2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        frag<AK>(sa, kb, t, wm + i * 16 + g, af[i][0], af[i][2]);
        frag<AK>(sa, kb, t, wm + i * 16 + 8 + g, af[i][1], af[i][3]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) frag<BKC>(sb, kb, t, wn + j * 8 + g, bf[j][0], bf[j][1]);
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) dmma(acc[i][j], af[i][0], af[i][1], af[i][2], af[i][3], bf[j][0], bf[j][1]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  const bool c_vec = ((ldc & 1) == 0) && (((uintptr_t)C & 15) == 0);
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int m = m0 + wm + i * 16 + h * 8 + g;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int n = n0 + wn + j * 8 + 2 * t;
          double* c = C + (long long)m * ldc + n;
          double v0 = alpha * acc[i][j][2 * h], v1 = alpha * acc[i][j][2 * h + 1];
          if (n + 1 < N) {
            if (beta) { v0 += c[0]; v1 += c[1]; }
            if (c_vec) *reinterpret_cast<double2*>(c) = make_double2(v0, v1);
            else { c[0] = v0; c[1] = v1; }
          } else if (n < N) {
            if (beta) v0 += c[0];
            c[0] = v0;
          }
        }
      }
    return;
  }
  // ---- a cluster adds its parts: every CTA leaves its tile in its own shared memory, then sums 64 / splits rows ----
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        *reinterpret_cast<double2*>(dsm + (wm + i * 16 + h * 8 + g) * DB + wn + j * 8 + 2 * t) =
            make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int rows = DB / splits;
  for (int q = threadIdx.x; q < rows * DB; q += DTHREADS) {
    const int r = rank * rows + q / DB, n = q % DB;
    const uint32_t local = smem_u32(dsm + r * DB + n);
    double v = 0.0;
    for (int p = 0; p < splits; p++) {
      uint32_t remote;
      double x;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(p));
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(remote) : "memory");
      v += x;
    }
    if (m0 + r < M && n0 + n < N) {
      double* c = C + (long long)(m0 + r) * ldc + n0 + n;
      *c = beta ? *c + alpha * v : alpha * v;
    }
  }
  // nobody leaves while a peer may still read its shared memory
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

thread_local int g_f64_splits = 0;      // 0: by the rule below

// CTAs per tile: K is cut while the CTAs stay within three per SM and a part keeps about a k-tile.  Measured, us for 1 | 2 | 4 |
// 8 parts: 64 x 64 x 2048 122 | 67 | 36 | 20; 362^3 25 | 19 | 14 | 12; 512^3 33 | 23 | 17 | 17; 100^3 9 | 11 | 7.5 | 5.8; and where
// the tiles fill the GPU, 1024^3 (256 tiles) 86 | 94 | 92 | 91, 2048^3 572 | 572 | 594 | 606.
int f64_splits(int M, int N, int K, int batch) {
  if (g_f64_splits) return g_f64_splits;
  const long long tiles = (long long)((M + DB - 1) / DB) * ((N + DB - 1) / DB) * batch;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= 3 * 148 && K / (2 * s) >= 12) s *= 2;
  return s;
}

template <bool AK, bool BKC>
int launch_f64(const void* A, const void* B, void* C, int M, int N, int K, int batch, long long lda, long long ldb, long long ldc,
               long long sA, long long sB, long long sC, double alpha, int beta, cudaStream_t s) {
  auto kern = gemm_f64_mma_kernel<AK, BKC>;
  GB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DSMEM));
  const int splits = f64_splits(M, N, K, batch);
  const int k_per = ((K + splits - 1) / splits + DBK - 1) / DBK * DBK;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)((long long)((M + DB - 1) / DB) * ((N + DB - 1) / DB) * splits), batch);
  cfg.blockDim = dim3(DTHREADS);
  cfg.dynamicSmemBytes = DSMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  GB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, (const double*)A, (const double*)B, (double*)C, M, N, K, lda, ldb, ldc, sA, sB, sC, alpha,
                                beta, splits, k_per));
  return gbh::E_OK;
}

// ---------------------------------------------------------------------------
// fp32 as three bf16 planes
// ---------------------------------------------------------------------------
// Plane p of the result holds the p-th bf16 part of src (rows, cols; row pitch ld): dst [3][rows][cols_p], cols_p = cols
// rounded up to 8, zero filled.  Bound by memory: 4 bytes read and 6 written per element; a thread turns eight
// neighbouring elements into three 16-byte stores.  (Six planes in the order of the products, two bytes at a time
// with a 64-bit division per element, took 267 us for the six operands of a 3000 x 1024 x 4096 layer; this takes 65.)
// An infinity or NaN stands in the lo plane, which meets the other operand's hi plane alone, so that no product with a
// lo or mid part of the other sign turns it into NaN; the hi plane holds +-1 in its place, with which an infinity of the other
// operand gets its sign.  (In the hi plane an infinity times an ordinary row gave NaN.)  A finite value that would round
// to infinity in bf16 is cut to bf16's largest value and keeps the rest in the other planes.
struct SplitArgs {
  const float* src;
  __nv_bfloat16* dst;
  int rows, cols, cols_p, vec, batch;
  long long ld, src_batch;
};
template <bool GUARD>
__device__ __forceinline__ void split3(const SplitArgs& a, int z, unsigned& most, unsigned& least) {
  const float* src = a.src + (long long)z * a.src_batch;
  const long long plane = (long long)a.rows * a.cols_p;
  __nv_bfloat16* dst = a.dst + (long long)z * 3 * plane;
  const int per_row = a.cols_p / 8;
  const unsigned total = (unsigned)a.rows * (unsigned)per_row;      // < 2^31: the operands' 16-bit planes fit 4 GiB
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned r = i / (unsigned)per_row;
    const int c = (int)(i - r * per_row) * 8;
    const float* s = src + (long long)r * a.ld + c;
    float x[8];
    if (a.vec && c + 8 <= a.cols) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(s)), v = __ldg(reinterpret_cast<const float4*>(s) + 1);
      x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] = c + j < a.cols ? __ldg(s + j) : 0.f;
    }
    __align__(16) __nv_bfloat16 pl[3][8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const bool fin = isfinite(x[j]);
      const float top = __uint_as_float(0x7f7f0000u);                 // bf16's largest value
      pl[0][j] = __float2bfloat16_rn(fin ? fminf(fmaxf(x[j], -top), top) : copysignf(1.f, x[j]));
      const float r1 = fin ? x[j] - __bfloat162float(pl[0][j]) : 0.f;
      pl[1][j] = __float2bfloat16_rn(r1);
      pl[2][j] = __float2bfloat16_rn(fin ? r1 - __bfloat162float(pl[1][j]) : x[j]);
      if (GUARD) {
        const unsigned u = __float_as_uint(x[j]) & 0x7fffffffu;
        most = max(most, u);
        least = max(least, 0u - u);
      }
    }
    __nv_bfloat16* d = dst + (long long)r * a.cols_p + c;
#pragma unroll
    for (int p = 0; p < 3; p++) *reinterpret_cast<uint4*>(d + p * plane) = *reinterpret_cast<const uint4*>(pl[p]);
  }
}
__global__ void __launch_bounds__(256) split3_kernel(const SplitArgs a) {
  unsigned most = 0u, least = 0u;
  split3<false>(a, blockIdx.z, most, least);
}

// Both operands of a product in one launch (blockIdx.y), and into guard[2 y] and [2 y + 1] the largest magnitude and minus the smallest
// one that is not zero, as bits (see planes_hold).
__global__ void __launch_bounds__(256) split3_both_kernel(const SplitArgs a, const SplitArgs b, unsigned* guard) {
  __shared__ unsigned sm[2][8];
  if ((int)blockIdx.z >= (blockIdx.y == 0 ? a.batch : b.batch)) return;
  unsigned most = 0u, least = 0u;
  if (blockIdx.y == 0) split3<true>(a, blockIdx.z, most, least);
  else split3<true>(b, blockIdx.z, most, least);
  most = __reduce_max_sync(0xffffffffu, most);
  least = __reduce_max_sync(0xffffffffu, least);
  if ((threadIdx.x & 31) == 0) {
    sm[0][threadIdx.x >> 5] = most;
    sm[1][threadIdx.x >> 5] = least;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned v = 0u, *word = guard + 2 * blockIdx.y + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 8; i++) v = max(v, sm[threadIdx.x][i]);
    if (v > *(volatile unsigned*)word) atomicMax(word, v);     // (few blocks raise it)
  }
}

}  // namespace

// CTAs that share a tile of the fp64 product: 1, 2, 4 or 8, 0 = chosen by size (for measurements and tests).
GB_EXPORT int gb_gemm_f64_tune(int splits) {
  if (splits != 0 && splits != 1 && splits != 2 && splits != 4 && splits != 8) {
    gbh::set_error("gb_gemm_f64_tune: splits is 0, 1, 2, 4 or 8");
    return gbh::E_BAD_ARG;
  }
  g_f64_splits = splits;
  return gbh::E_OK;
}

// C = alpha * op(A) op(B) (+ C) in float64 on the double-precision tensor cores.
GB_EXPORT int gb_gemm_f64(const void* A, const void* B, void* C, int M, int N, int K, int batch, int transA,
                          int transB, long long lda, long long ldb, long long ldc, long long sA, long long sB,
                          long long sC, double alpha, int beta, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) {
    gbh::set_error("gb_gemm_f64: empty problem");
    return gbh::E_BAD_ARG;
  }
  if ((long long)((M + DB - 1) / DB) * ((N + DB - 1) / DB) >= (1LL << 28) || batch > 65535) {
    gbh::set_error("gb_gemm_f64: problem too large");
    return gbh::E_TOO_LARGE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (!transA && transB) return launch_f64<true, true>(A, B, C, M, N, K, batch, lda, ldb, ldc, sA, sB, sC, alpha, beta, st);
  if (!transA) return launch_f64<true, false>(A, B, C, M, N, K, batch, lda, ldb, ldc, sA, sB, sC, alpha, beta, st);
  if (transB) return launch_f64<false, true>(A, B, C, M, N, K, batch, lda, ldb, ldc, sA, sB, sC, alpha, beta, st);
  return launch_f64<false, false>(A, B, C, M, N, K, batch, lda, ldb, ldc, sA, sB, sC, alpha, beta, st);
}

// Bytes of scratch gb_gemm_f32x3 needs for the split operands.
GB_EXPORT long long gb_gemm_f32x3_workspace(int M, int N, int K, int batch) {
  const long long Kp = (K + 7) / 8 * 8, Mp = (M + 7) / 8 * 8, Np = (N + 7) / 8 * 8;
  const long long a = M * Kp > K * Mp ? M * Kp : K * Mp, b = N * Kp > K * Np ? N * Kp : K * Np;   // either storage form
  return 2LL * batch * 3 * (a + b) + 256;
}

// fp32 GEMM through three bf16 planes per operand (see the file header).  bias: fp32 [N] or null.  workspace:
// gb_gemm_f32x3_workspace() bytes; split_ws / split_ws_bytes: optional split-K scratch handed on to the bf16 GEMM.  chain: the most
// of K that one accumulator takes (a multiple of 64, with room for every slice in split_ws; 0: any length).  guarded: operands that
// could overflow between the planes, or whose parts would be subnormal, are multiplied by FMA instead; the splits find out, the plane
// kernels then do nothing, and the FMA kernel else.
GB_EXPORT int gb_gemm_f32x3(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int batch, int transA,
                            int transB, long long lda, long long ldb, long long ldc, long long sA, long long sB,
                            long long sC, float alpha, int beta, void* workspace, long long workspace_bytes,
                            void* split_ws, long long split_ws_bytes, int chain, int guarded, void* stream) {
  if (workspace == nullptr || workspace_bytes < gb_gemm_f32x3_workspace(M, N, K, batch)) {
    gbh::set_error("gb_gemm_f32x3: workspace too small");
    return gbh::E_BAD_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const bool share_a = batch > 1 && sA == 0, share_b = batch > 1 && sB == 0;
  // an operand as stored: (rows, cols)
  const int ar = transA ? K : M, ac = transA ? M : K, br = transB ? N : K, bc = transB ? K : N;
  const long long acp = (ac + 7) / 8 * 8, bcp = (bc + 7) / 8 * 8;
  const long long plane_a = ar * acp, plane_b = br * bcp;
  __nv_bfloat16* a3 = (__nv_bfloat16*)workspace;
  __nv_bfloat16* b3 = a3 + 3 * plane_a * (share_a ? 1 : batch);
  auto operand = [&](const void* src, __nv_bfloat16* dst, int rows, int cols, long long ld, long long cols_p, long long sb, int n) {
    return SplitArgs{(const float*)src, dst, rows, cols, (int)cols_p, (ld & 3) == 0 && (sb & 3) == 0 && (((uintptr_t)src) & 15) == 0, n, ld, sb};
  };
  auto blocks_of = [](const SplitArgs& o) {
    const long long blocks = (o.rows * (o.cols_p / 8ll) + 255) / 256;
    return (unsigned)(blocks < 148 * 16 ? blocks : 148 * 16);
  };
  const SplitArgs sa = operand(A, a3, ar, ac, lda, acp, sA, share_a ? 1 : batch), sb = operand(B, b3, br, bc, ldb, bcp, sB, share_b ? 1 : batch);
  unsigned* guard = nullptr;
  int top = 0;
  if (guarded) {
    guard = (unsigned*)(((uintptr_t)(b3 + 3 * plane_b * sb.batch) + 15) & ~(uintptr_t)15);   // (256 bytes of the workspace are left over)
    // so far the products and their sums (of fewer than 2^26) stay finite, and what alpha makes of them
    top = 100 - (fabsf(alpha) > 1.f ? ilogbf(alpha) : 0);
    GB_CUDA_OK(cudaMemsetAsync(guard, 0, 16, s));
    const unsigned most = blocks_of(sa) > blocks_of(sb) ? blocks_of(sa) : blocks_of(sb);
    split3_both_kernel<<<dim3(most, 2, sa.batch > sb.batch ? sa.batch : sb.batch), 256, 0, s>>>(sa, sb, guard);
  } else {
    split3_kernel<<<dim3(blocks_of(sa), 1, sa.batch), 256, 0, s>>>(sa);
    split3_kernel<<<dim3(blocks_of(sb), 1, sb.batch), 256, 0, s>>>(sb);
  }
  GB_CUDA_OK(cudaGetLastError());
  // Planes 0, 1, 2 = hi, mid, lo.  One launch and one accumulator for all six products, from the smallest to the largest:
  // lo hi, hi lo, mid mid, then mid hi, hi mid, then hi hi.  The tensor core truncates each sum at its accumulator's last
  // bit, so the small products must be in before the large ones; the error is then that of the hi hi chain alone
  // (relative to 64 bits at 3000 x 4096 x 1024: 1.0e-6 in this order in one accumulator, in two and in three).
  // A slice of a split K runs all six products over its part of K, which shortens that chain.
  const int rc = gemm_bf16_planes(a3, b3, (float*)C, (const float*)bias, M, N, K, batch, transA, transB, acp, bcp, ldc, plane_a, plane_b,
                                  share_a, share_b, sC, 6, 0x001102u, 0x010120u, alpha, beta, split_ws, split_ws_bytes, s, chain, guard, top);
  if (rc || guard == nullptr) return rc;
  return gemm_fma_unless_planes(A, B, (float*)C, (const float*)bias, M, N, K, batch, transA, transB, lda, ldb, ldc, sA, sB, sC, alpha, beta,
                                guard, top, s);
}

// ---------------------------------------------------------------------------
// in-library benchmark loops (milliseconds per call; -1 on an allocation failure)
// ---------------------------------------------------------------------------
namespace {
template <typename F>
double bench_loop(int iters, F&& fn) {
  for (int i = 0; i < 5; i++)
    if (fn() != 0) return -2.0;
  if (cudaDeviceSynchronize() != cudaSuccess) return -2.0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0);
  for (int i = 0; i < iters; i++) fn();
  cudaEventRecord(e1);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return (double)ms / iters;
}
}  // namespace

// Resident (m,k) @ (k,n).  dtype: 0 bf16, 1 fp16 (tcgen05, fp32 accumulate, operand bytes zeroed
// like the reference's fp16 loop), 2 fp32 (three-plane path), 3 fp64 (tensor-core fp64); the
// fp32 / fp64 operand bytes are set to 0x01 like the reference's loop.
GB_EXPORT double gb_bench_matmul(int m, int k, int n, int iters, int dtype) {
  const size_t esz = dtype == DT_F64 ? 8 : (dtype == DT_F32 ? 4 : 2);
  void *A = nullptr, *B = nullptr, *C = nullptr, *ws = nullptr;
  if (cudaMalloc(&A, esz * (size_t)m * k) != cudaSuccess) return -1.0;
  if (cudaMalloc(&B, esz * (size_t)k * n) != cudaSuccess) { cudaFree(A); return -1.0; }
  if (cudaMalloc(&C, esz * (size_t)m * n) != cudaSuccess) { cudaFree(A); cudaFree(B); return -1.0; }
  const int fill = esz == 2 ? 0 : 1;
  cudaMemset(A, fill, esz * (size_t)m * k);
  cudaMemset(B, fill, esz * (size_t)k * n);
  long long ws_bytes = 0;
  if (dtype == DT_F32) {
    ws_bytes = gb_gemm_f32x3_workspace(m, n, k, 1);
    if (cudaMalloc(&ws, ws_bytes) != cudaSuccess) { cudaFree(A); cudaFree(B); cudaFree(C); return -1.0; }
  }
  double ms;
  if (dtype == DT_F64)
    ms = bench_loop(iters, [&] { return gb_gemm_f64(A, B, C, m, n, k, 1, 0, 0, k, n, n, 0, 0, 0, 1.0, 0, nullptr); });
  else if (dtype == DT_F32)
    ms = bench_loop(iters, [&] {
      return gb_gemm_f32x3(A, B, C, nullptr, m, n, k, 1, 0, 0, k, n, n, 0, 0, 0, 1.f, 0, ws, ws_bytes, nullptr, 0, 0, 0, nullptr);
    });
  else
    ms = bench_loop(iters, [&] {
      return gb_gemm16(A, B, C, nullptr, 0, nullptr, m, n, k, 1, 0, 0, k, n, n, 0, 0, 0, 0, 0, dtype, dtype, 0, 0, 0,
                       1.f, 0, nullptr, 0, nullptr);
    });
  cudaFree(A); cudaFree(B); cudaFree(C);
  if (ws) cudaFree(ws);
  return ms;
}

// Resident elementwise add of n elements (f32 != 0: float, else double).
GB_EXPORT double gb_bench_add(long long n, int iters, int f32) {
  const size_t esz = f32 ? 4 : 8;
  void *A = nullptr, *B = nullptr, *C = nullptr;
  if (cudaMalloc(&A, esz * n) != cudaSuccess) return -1.0;
  if (cudaMalloc(&B, esz * n) != cudaSuccess) { cudaFree(A); return -1.0; }
  if (cudaMalloc(&C, esz * n) != cudaSuccess) { cudaFree(A); cudaFree(B); return -1.0; }
  cudaMemset(A, 1, esz * n);
  cudaMemset(B, 1, esz * n);
  const double ms = bench_loop(iters, [&] { return gb_binary(0, f32 ? DT_F32 : DT_F64, A, B, C, n, 0, nullptr, nullptr, nullptr, nullptr); });
  cudaFree(A); cudaFree(B); cudaFree(C);
  return ms;
}

// Resident attention forward over (BH, S, d) in bf16 (d = 64 or 128), zero-filled like the reference's loop.
GB_EXPORT double gb_bench_flash_attn(int BH, int S, int d, int iters, int causal) {
  const size_t n = (size_t)BH * S * d;
  void *Q = nullptr, *K = nullptr, *V = nullptr, *O = nullptr;
  float* L = nullptr;
  if (cudaMalloc(&Q, 2 * n) != cudaSuccess) return -1.0;
  if (cudaMalloc(&K, 2 * n) != cudaSuccess) { cudaFree(Q); return -1.0; }
  if (cudaMalloc(&V, 2 * n) != cudaSuccess) { cudaFree(Q); cudaFree(K); return -1.0; }
  if (cudaMalloc(&O, 2 * n) != cudaSuccess) { cudaFree(Q); cudaFree(K); cudaFree(V); return -1.0; }
  if (cudaMalloc(&L, 4 * (size_t)BH * S) != cudaSuccess) { cudaFree(Q); cudaFree(K); cudaFree(V); cudaFree(O); return -1.0; }
  cudaMemset(Q, 0, 2 * n);
  cudaMemset(K, 0, 2 * n);
  cudaMemset(V, 0, 2 * n);
  // (BH, S, d) read as batch 1, BH heads: head stride S * d, sequence stride d
  const long long sb = (long long)n, ss = d, sh = (long long)S * d;
  const float scale = 1.f / sqrtf((float)d);
  const double ms = bench_loop(iters, [&] {
    return gb_flash_fwd(DT_BF16, Q, K, V, O, L, 1, BH, S, S, d, sb, ss, sh, sb, ss, sh, sb, ss, sh, sb, ss, sh, scale,
                        causal, nullptr);
  });
  cudaFree(Q); cudaFree(K); cudaFree(V); cudaFree(O); cudaFree(L);
  return ms;
}
