// Implicit-GEMM convolution on tcgen05: forward, data gradient and weight gradient without an
// im2col matrix in memory.
//
// The reference computes a convolution as a dense 0/1 gather-matrix product that materialises
// the (N, L, C*T) column tensor, then a batched MatMul (nn/conv.go:341-380, nn/gather.go:99-181),
// and lets autograd differentiate those tape nodes.  Here the column tensor never exists: the
// producer warps of each CTA gather the operand tiles straight from the (N, C, spatial) tensors
// into the 128-byte-swizzled shared-memory layout that tcgen05.mma reads (through the same
// int32 window index map the pooling and fold kernels use: entry [l][tap] is the source position
// of tap `tap` of output position `l`, or -1 for padding), one elected thread issues the MMAs into
// a 128 x 128 fp32 accumulator in tensor memory, and the same warps run the epilogue.
//
//   forward   y[n][co][l]  = bias[co] + sum_{c,tap} W[co][c][tap] * x[n][c][idx[l][tap]]
//             GEMM per image: M = C_out, N = L, K = C_in * T; A = weights, B = gathered windows.
//   dgrad     the same kernel with x := dy, idx := the inverse map ([s][tap] -> l or -1) and the
//             weights regrouped as a (C_in, C_out * T) matrix.
//   wgrad     dW[co][(c,tap)] = sum_{n,l} dy[n][co][l] * x[n][c][idx[l][tap]]
//             ONE GEMM over the whole batch: M = C_out, N = C_in * T, K = N_img * L, split over
//             CTAs along K into fp32 partials that a second kernel adds in split order
//             (deterministic).
//
// No tensor map is involved (every operand is gathered with ordinary loads from this GPU's own
// memory), so the kernels may run inside multi-GPU jobs.  Every wait is bounded.
#include "conv.cuh"

using namespace gb;
using gbc::float_to_raw16;
using gbc::raw16_to_float;

namespace {

constexpr int CBM = 128, CBN = 128, CBK = 64, CSTAGES = 2;
constexpr int CA_BYTES = CBM * CBK * 2, CB_BYTES = CBN * CBK * 2, CSTAGE_BYTES = CA_BYTES + CB_BYTES;
constexpr int CPRODUCERS = 256;            // threads 0..127 fill A rows, 128..255 fill B rows
constexpr int CTHREADS = CPRODUCERS + 32;  // + the MMA warp
constexpr int CMAX_T_SMEM = 32;            // window taps up to which the forward stages its index rows
constexpr int CSMEM = CSTAGES * CSTAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/ + CBN * CMAX_T_SMEM * 4;

struct ConvArgs {
  // forward / dgrad
  const uint16_t* W;       // (M, K) row-major weights, K = C * T ordered (c, tap)
  int w_vec;               // rows may be read in 16-byte pieces (K % 8 == 0 and an aligned base)
  const int2* ktab;        // [K rounded up to 128]: {c * S, tap} for k < K, {-1, 0} beyond
  const uint16_t* X;       // (Nimg, C, S): the tensor whose windows are gathered
  const int* idx;          // [L][T]
  void* Y;                 // forward / dgrad: (Nimg, M, L) 16-bit; wgrad: fp32 partials [splits][M][KK]
  const uint16_t* bias;    // [M], same 16-bit type, or null
  // wgrad
  const uint16_t* DY;      // (Nimg, M, L)
  int Nimg, C, S, L, T, M;
  int bf16;
  long long r_per_split;   // wgrad: contraction indices per split (multiple of 64)
  int* status;
};

// One 16-byte chunk (8 consecutive k) into row `row`, chunk `c8` of a K-major 128-byte-swizzled tile.
__device__ __forceinline__ void store_chunk(uint8_t* tile, int row, int c8, const uint16_t (&v)[8]) {
  uint4 u;
  u.x = (uint32_t)v[0] | ((uint32_t)v[1] << 16);
  u.y = (uint32_t)v[2] | ((uint32_t)v[3] << 16);
  u.z = (uint32_t)v[4] | ((uint32_t)v[5] << 16);
  u.w = (uint32_t)v[6] | ((uint32_t)v[7] << 16);
  *reinterpret_cast<uint4*>(tile + row * 128 + ((c8 ^ (row & 7)) << 4)) = u;
}

// MODE 0: forward / dgrad (grid: L tiles, M tiles, images); MODE 1: wgrad (grid: KK tiles, M tiles, splits)
template <int MODE>
__global__ void __launch_bounds__(CTHREADS, 2)
conv_igemm_kernel(const ConvArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + CSTAGES * CSTAGE_BYTES);
  uint64_t* full_bar = bars;              // [CSTAGES], 8 arrivals: one per producer warp
  uint64_t* empty_bar = bars + CSTAGES;   // [CSTAGES], 1 arrival: tcgen05.commit
  uint64_t* done_bar = bars + 2 * CSTAGES;
  uint32_t* tmem_slot = (uint32_t*)(done_bar + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = a.C * a.T;

  if (threadIdx.x == 0) {
    for (int s = 0; s < CSTAGES; s++) { mbar_init(&full_bar[s], CPRODUCERS / 32); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, CBN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // contraction range of this CTA, in k-blocks of 64
  long long kc_begin, kc_end;   // element indices along the contraction
  if (MODE == 0) {
    kc_begin = 0;
    kc_end = K;
  } else {
    const long long R = (long long)a.Nimg * a.L;
    kc_begin = (long long)blockIdx.z * a.r_per_split;
    kc_end = kc_begin + a.r_per_split < R ? kc_begin + a.r_per_split : R;
  }
  const int nkb = kc_end > kc_begin ? (int)((kc_end - kc_begin + CBK - 1) / CBK) : 0;
  const int m0 = blockIdx.y * CBM, n0 = blockIdx.x * CBN;

  if (warp < 8) {
    // ---------------- producers ----------------
    // Warps 0-3 fill the A tile, warps 4-7 the B tile, 32 rows each.  The kernel is bound by the
    // instructions of these gathers, so they are kept to a handful per element: the split of a
    // contraction index k into (channel offset, tap) comes from a table built once per geometry
    // (ktab[k] = {c * S, tap}, {-1, 0} past the end), window index rows are staged in shared
    // memory, offsets are 32-bit, and every load is unconditional (offset 0 when the element is
    // padding, the value zeroed afterwards) so that many are in flight per thread.
    const bool is_a = warp < 4;
    const int wq = warp & 3;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const int e0 = 2 * lane;
    int* sidx = reinterpret_cast<int*>(smem + CSTAGES * CSTAGE_BYTES + 256);   // [128][T] (fwd) or [64][T] (wgrad)
    // Forward / dgrad tiles run over the positions of ALL images (p = image * L + l), so a plane whose
    // size is not a multiple of the tile (13 x 13 = 169) does not leave a mostly empty second tile per image.
    const long long P = (long long)a.Nimg * a.L;
    if (MODE == 0 && !is_a) {
      // the index rows of this CTA's 128 positions, staged once
      const int total = CBN * a.T;
      for (int i = threadIdx.x - CBM; i < total; i += CBN) {
        const long long pp = (long long)n0 + i / a.T;
        sidx[i] = pp < P ? __ldg(a.idx + (pp % a.L) * a.T + i % a.T) : -1;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");   // the four B warps only
    }
    for (int kb = 0; kb < nkb && ok; kb++) {
      if (lane == 0) ok = mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, a.status, ST_CONV_TIMEOUT, 1);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      uint8_t* tile = smem + stage * CSTAGE_BYTES + (is_a ? 0 : CA_BYTES);
      const long long k0 = kc_begin + (long long)kb * CBK;
      if (MODE == 0 && is_a) {
        // weights as a row-major (M, K) matrix: thread = row
        const int row = threadIdx.x;
        const int m = m0 + row;
        const uint16_t* wr = a.W + (long long)(m < a.M ? m : a.M - 1) * K;
        if (a.w_vec) {
#pragma unroll
          for (int c8 = 0; c8 < 8; c8++) {
            const int k = (int)k0 + c8 * 8;
            uint4 u = make_uint4(0u, 0u, 0u, 0u);
            if (m < a.M && k < K) u = __ldg(reinterpret_cast<const uint4*>(wr + k));   // K % 8 == 0: whole chunks
            *reinterpret_cast<uint4*>(tile + row * 128 + ((c8 ^ (row & 7)) << 4)) = u;
          }
        } else {
#pragma unroll 1
          for (int h = 0; h < 4; h++) {
            uint16_t v[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
              const int k = (int)k0 + h * 16 + j;
              v[j] = __ldg(wr + (k < K ? k : K - 1));
              if (!(m < a.M && k < K)) v[j] = 0;
            }
            store_chunk(tile, row, 2 * h, *reinterpret_cast<const uint16_t(*)[8]>(&v[0]));
            store_chunk(tile, row, 2 * h + 1, *reinterpret_cast<const uint16_t(*)[8]>(&v[8]));
          }
        }
      } else if (MODE == 0) {
        // window operand, lanes along positions: consecutive positions read consecutive elements
        const int row = wq * 32 + lane;
        const int* ir = sidx + row * a.T;
        const long long pp = (long long)n0 + row;
        const uint16_t* xn = a.X + (pp < P ? pp / a.L : 0) * a.C * a.S;   // this row's image (padding rows read image 0, zeroed)
        const int2* kt = a.ktab + k0;
#pragma unroll 1
        for (int h = 0; h < 4; h++) {
          int off[16];
          uint16_t v[16];
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const int2 t = __ldg(kt + h * 16 + j);       // the same entry for the whole warp
            const int src = ir[t.y];
            off[j] = (t.x >= 0 && src >= 0) ? t.x + src : -1;
          }
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = __ldg(xn + (off[j] >= 0 ? off[j] : 0));
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = off[j] >= 0 ? v[j] : (uint16_t)0;
          store_chunk(tile, row, 2 * h, *reinterpret_cast<const uint16_t(*)[8]>(&v[0]));
          store_chunk(tile, row, 2 * h + 1, *reinterpret_cast<const uint16_t(*)[8]>(&v[8]));
        }
      } else {
        // weight gradient: lanes along the contraction index r = image * L + l
        int nn[2], ll[2];
        bool kv[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const long long r = k0 + e0 + e;
          kv[e] = r < kc_end;
          const long long rc = kv[e] ? r : kc_end - 1;
          nn[e] = (int)(rc / a.L);
          ll[e] = (int)(rc % a.L);
        }
        if (!is_a) {
          // index rows of this k-block's 64 positions: [64][T]
          asm volatile("bar.sync 1, 128;" ::: "memory");   // the previous k-block's readers are done
          const int total = CBK * a.T;
          for (int i = threadIdx.x - CBM; i < total; i += CBN) {
            const long long r = k0 + i / a.T;
            sidx[i] = r < kc_end ? __ldg(a.idx + (r % a.L) * a.T + i % a.T) : -1;
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        const uint16_t* b0 = is_a ? a.DY + ((long long)nn[0] * a.M) * a.L + ll[0] : a.X + (long long)nn[0] * a.C * a.S;
        const uint16_t* b1 = is_a ? a.DY + ((long long)nn[1] * a.M) * a.L + ll[1] : a.X + (long long)nn[1] * a.C * a.S;
#pragma unroll 1
        for (int rb = 0; rb < 32; rb += 8) {
          uint16_t v[8][2];
          int o0[8], o1[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int rowi = wq * 32 + rb + j;
            if (is_a) {
              const int m = m0 + rowi;
              o0[j] = o1[j] = m < a.M ? m * a.L : -1;
            } else {
              const int kk = n0 + rowi;
              const int2 t = __ldg(a.ktab + kk);           // ktab covers K rounded up to 128
              const int s0 = sidx[e0 * a.T + t.y], s1 = sidx[(e0 + 1) * a.T + t.y];
              o0[j] = (t.x >= 0 && s0 >= 0) ? t.x + s0 : -1;
              o1[j] = (t.x >= 0 && s1 >= 0) ? t.x + s1 : -1;
            }
          }
#pragma unroll
          for (int j = 0; j < 8; j++) {
            v[j][0] = __ldg(b0 + (o0[j] >= 0 ? o0[j] : 0));
            v[j][1] = __ldg(b1 + (o1[j] >= 0 ? o1[j] : 0));
          }
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int rowi = wq * 32 + rb + j;
            const uint32_t lo = (o0[j] >= 0 && kv[0]) ? v[j][0] : 0u, hi = (o1[j] >= 0 && kv[1]) ? v[j][1] : 0u;
            uint8_t* d = tile + rowi * 128 + ((((e0 >> 3) ^ (rowi & 7))) << 4) + (e0 & 7) * 2;
            *reinterpret_cast<uint32_t*>(d) = lo | (hi << 16);
          }
        }
      }
      fence_proxy_async_smem();   // generic-proxy writes become visible to the tensor core
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[stage]);
      if (++stage == CSTAGES) { stage = 0; phase ^= 1; }
    }
  } else if (elect_one()) {
    // ---------------- MMA issuer (one thread) ----------------
    uint32_t id = make_idesc(1u, 0u, false, false, CBM, CBN);
    if (a.bf16) id |= (1u << 7) | (1u << 10);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = 0; kb < nkb && ok; kb++) {
      ok = mbar_wait(&full_bar[stage], phase, abort_flag, a.status, ST_CONV_TIMEOUT, 2);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sa = smem_u32(smem + stage * CSTAGE_BYTES);
      const uint32_t sb = sa + CA_BYTES;
#pragma unroll
      for (int k = 0; k < CBK / 16; k++) {
        // K-major tiles: 8-row groups 1024 B apart, one MMA step is 32 B along K
        tc_mma_f16(tmem_base, make_smem_desc_sw128(sa + k * 32, 16, 1024), make_smem_desc_sw128(sb + k * 32, 16, 1024),
                   id, (kb > 0) || k != 0);
      }
      tc_commit(&empty_bar[stage]);
      if (++stage == CSTAGES) { stage = 0; phase ^= 1; }
    }
    tc_commit(done_bar);   // arrives when every MMA above has finished (at once if there were none)
  }

  // ---------------- epilogue: the eight producer warps ----------------
  // tcgen05.ld gives a thread one accumulator row (lane = row).  Rows of the outputs are far
  // apart in memory, so each warp turns its 32 x 32 block around through shared memory (the
  // ring is idle by now) and stores with lanes along the contiguous dimension.
  if (warp < 8) {
    bool ok = true;
    if (lane == 0) ok = mbar_wait(done_bar, 0, abort_flag, a.status, ST_CONV_TIMEOUT, 3);
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    if (ok) {
      tc_fence_after();
      const int q = warp & 3, half = warp >> 2;        // TMEM lane quarter, column half
      const int mrow0 = m0 + q * 32;
      float* stf = reinterpret_cast<float*>(smem + warp * (32 * 33 * 4));   // [32][33] floats per warp
#pragma unroll 1
      for (int cc = 0; cc < 2; cc++) {
        const int col0 = half * 64 + cc * 32;
        uint32_t r[32];
        if (nkb > 0) {
          tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + col0, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; j++) r[j] = 0u;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; j++) stf[lane * 33 + j] = __uint_as_float(r[j]);
        __syncwarp();
        const int col = n0 + col0 + lane;
        if (MODE == 0) {
          const long long pp = (long long)n0 + col0 + lane;          // position over all images
          const bool live = pp < (long long)a.Nimg * a.L;
          const long long img = live ? pp / a.L : 0;
          const int lpos = (int)(pp - img * a.L);
          uint16_t* yb = (uint16_t*)a.Y + img * a.M * a.L + lpos;
          for (int rr = 0; rr < 32; rr++) {
            const int m = mrow0 + rr;
            if (m >= a.M) break;
            if (live) {
              const float bv = a.bias ? raw16_to_float(__ldg(a.bias + m), a.bf16) : 0.f;
              const float v = stf[rr * 33 + lane] + bv;
              yb[(long long)m * a.L] =
                  a.bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
            }
          }
        } else {
          float* pb = (float*)a.Y + (long long)blockIdx.z * a.M * K;
          for (int rr = 0; rr < 32; rr++) {
            const int m = mrow0 + rr;
            if (m >= a.M) break;
            if (col < K) pb[(long long)m * K + col] = stf[rr * 33 + lane];
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem_base, CBN);
}

// dW[m][c * T + tap] = (beta ? dW : 0) + sum_s part[s][m][kk], kk = (tap, c) when tap_major, else (c, tap).  A block
// owns 32 consecutive elements; its eight warps add every eighth split and their sums are added in warp order
// (deterministic).  One thread per element walked all splits alone: 9 us for 296 splits of 1728 elements.
__global__ void __launch_bounds__(256) conv_wgrad_finish_kernel(const float* __restrict__ part, uint16_t* __restrict__ dW,
                                                                long long n, int C, int T, int splits, int bf16, int beta,
                                                                int tap_major) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sm[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (long long b = blockIdx.x; b * 32 < n; b += gridDim.x) {
    const long long i = b * 32 + lane;
    float s = 0.f;
    if (i < n) {
#pragma unroll 4
      for (int sp = warp; sp < splits; sp += 8) s += part[(long long)sp * n + i];
    }
    sm[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && i < n) {
      const int K = C * T;
      const long long m = i / K;
      const int kk = (int)(i - m * K), tap = kk / C;
      uint16_t* d = dW + (tap_major ? m * K + (long long)(kk - tap * C) * T + tap : i);
      s = beta ? raw16_to_float(*d, bf16) : 0.f;
#pragma unroll
      for (int w = 0; w < 8; w++) s += sm[w][lane];
      *d = float_to_raw16(s, bf16);
    }
    __syncthreads();
  }
}

// Convolutions with a short contraction (C * T <= 32: the first layer of an image network, 3 channels x 3 x 3).
// A tcgen05 tile would spend its time on set-up and an fp32 loop per position on its multiply-adds and their
// weight reads (57 us forward, 97 us weight gradient at 256 x 64 channels x 900 positions); the contraction is
// two k-steps of the warp-level mma.sync m16n8k16:
//  * a warp takes 32 consecutive positions of the flattened batch; the index rows of those positions are
//    contiguous in the map, so they are copied to shared memory with coalesced loads, and lane p gathers the K
//    inputs of position p (neighbouring lanes, neighbouring addresses) into shared memory, from which the
//    fragments are read.  Gathering the fragments directly cost eight sectors a load (43 and 55 us);
//  * column n = 2t + e of n-tile j stands for position 8t + 2j + e, so a lane's results of the four n-tiles are eight
//    consecutive positions of a channel (V of them at a time are aligned when V divides L).
// Forward 23 us, weight gradient 35 us; bound by the gathers and the 29.5 MB of outputs or gradients.
constexpr int kDirectK = 32;
constexpr int kSmallWarps = 8;
constexpr int kSmallSmem = 96 * 1024;   // limit of the dynamic shared memory: windows of 32 taps alone take 49 KB

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], int bf16) {
  if (bf16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Position p0 of a warp's 32 as (image, position in the image).  The first ones are below 2^31 (148 * 8 CTAs of 256), and so are the
// strides from one to the next: no 64-bit division.
struct SmallPos {
  int img;
  unsigned l;
  __device__ __forceinline__ SmallPos(unsigned p, unsigned L) : img((int)(p / L)), l(p % L) {}
  __device__ __forceinline__ void advance(const SmallPos& by, unsigned L) {
    img += by.img;
    l += by.l;
    if (l >= L) { l -= L; img++; }
  }
};

// Index rows of the 32 positions from `at` on into si[32 * T]: rows of consecutive positions follow one another, from the
// end of an image's map to its beginning.  img, l: this lane's position.
__device__ __forceinline__ void stage_index(int* si, const int* __restrict__ idx, const SmallPos& at, unsigned L, int T, int& img, unsigned& l) {
  const int lane = threadIdx.x & 31;
  const long long LT = (long long)L * T;
  __syncwarp();
  for (int j0 = 0; j0 < T; j0 += 8) {                      // eight loads in flight: one at a time, T load latencies in a row
    int v[8];
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j0 + j < T) {
        long long f = (long long)at.l * T + (j0 + j) * 32 + lane;
        if (f >= LT) {                                     // past the end by less than 32 T <= 1024
          const unsigned past = (unsigned)(f - LT);
          f = past < LT ? past : past % (unsigned)LT;
        }
        v[j] = __ldg(idx + f);
      }
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j0 + j < T) si[(j0 + j) * 32 + lane] = v[j];
  }
  l = at.l + lane;
  img = at.img;
  while (l >= L) { l -= L; img++; }
  __syncwarp();
}

// The 32 (K of them real) inputs of this lane's position, two at a time, to put(k, v[k], v[k + 1]); image img, index rows si.  B
// loads are in flight together: put writes shared memory, past which the compiler moves no later index read (64 images, 3 x
// 31 x 31 to 64 channels, forward 28.3 -> 10.5 us with this, the batched index rows and the wide stores below).
template <int B, typename F>
__device__ __forceinline__ void gather_windows(const uint16_t* __restrict__ x, int img, bool live, const int* si, int C, int S, int T,
                                               const F& put) {
  const int K = C * T;
  const uint16_t* xc = x + (live ? (long long)img * C * S : 0);
  const int* row = si + (threadIdx.x & 31) * T;
  int tap = 0;
#pragma unroll
  for (int k0 = 0; k0 < kDirectK; k0 += B) {
    uint32_t v[B];
#pragma unroll
    for (int e = 0; e < B; e++) {
      v[e] = 0u;
      if (k0 + e < K) {
        const int src = row[tap];
        if (live && src >= 0) v[e] = __ldg(xc + src);
        if (++tap == T) { tap = 0; xc += S; }
      }
    }
#pragma unroll
    for (int e = 0; e < B; e += 2) put(k0 + e, v[e], v[e + 1]);
  }
  __syncwarp();
}

// Where the runs of V of the eight consecutive positions from `at` + 8t on start in a (Nimg, M, L) tensor (channel 0), -1 past
// the end.  V divides L, so a run never straddles images or the end.
template <int V>
__device__ __forceinline__ void run_starts(long long (&start)[8 / V], const SmallPos& at, int t, int Nimg, int M, unsigned L) {
  unsigned l = at.l + 8 * t;
  int img = at.img;
  while (l >= L) { l -= L; img++; }
#pragma unroll
  for (int i = 0; i < 8 / V; i++) {
    start[i] = img < Nimg ? (long long)img * M * L + l : -1;
    l += V;
    if (l >= L) { l -= L; img++; }
  }
}
// Eight values of a channel (row offset m * L), V at a time.
template <int V>
__device__ __forceinline__ void store8(uint16_t* __restrict__ y, const uint32_t (&v)[4], const long long (&at)[8 / V]) {
#pragma unroll
  for (int i = 0; i < 8 / V; i++) {
    if (at[i] < 0) return;
    uint16_t* d = y + at[i];
    if constexpr (V == 8) *reinterpret_cast<uint4*>(d) = make_uint4(v[0], v[1], v[2], v[3]);
    else if constexpr (V == 4) *reinterpret_cast<uint2*>(d) = make_uint2(v[2 * i], v[2 * i + 1]);
    else if constexpr (V == 2) *reinterpret_cast<uint32_t*>(d) = v[i];
    else *d = (uint16_t)(v[i / 2] >> (16 * (i & 1)));
  }
}
template <int V>
__device__ __forceinline__ void load8(const uint16_t* __restrict__ y, uint32_t (&v)[4], const long long (&at)[8 / V]) {
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = 0u;
#pragma unroll
  for (int i = 0; i < 8 / V; i++) {
    if (at[i] < 0) return;
    const uint16_t* d = y + at[i];
    if constexpr (V == 8) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(d));
      v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
    } else if constexpr (V == 4) {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(d));
      v[2 * i] = u.x; v[2 * i + 1] = u.y;
    } else if constexpr (V == 2) {
      v[i] = __ldg(reinterpret_cast<const uint32_t*>(d));
    } else {
      v[i / 2] |= (uint32_t)__ldg(d) << (16 * (i & 1));
    }
  }
}

// y[n][m][l] = bias[m] + sum_k w[m][k] x[n][c(k)][idx[l][tap(k)]]: A = weights (16 channels x 16 k), B = windows (16 k x 8
// positions).  The weights sit in shared memory in fragment order.
template <int V>
__global__ void __launch_bounds__(kSmallWarps * 32)
conv_direct_small_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, const int* __restrict__ idx,
                         const uint16_t* __restrict__ bias, uint16_t* __restrict__ y, int Nimg, int C, int S, int L, int T,
                         int M, int bf16) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) uint32_t dsm[];
  const int MT = (M + 15) / 16, K = C * T;
  uint32_t* wf = dsm;                                    // [MT][2 k-steps][32 lanes][4]
  float* sbias = reinterpret_cast<float*>(wf + MT * 256);   // [MT * 16]
  int* si = reinterpret_cast<int*>(sbias + MT * 16) + (threadIdx.x >> 5) * 32 * (T + 17);
  uint32_t* sp = reinterpret_cast<uint32_t*>(si + 32 * T);   // [32 positions][16 pairs of k], pitch 17
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const unsigned first = (blockIdx.x * kSmallWarps + (threadIdx.x >> 5)) * 32u, stride = gridDim.x * kSmallWarps * 32u;
  SmallPos at(first, L);
  const SmallPos by(stride, L);
  int img;
  unsigned l;
  auto fetch = [&]() {                                     // index rows and windows of the warp's positions into sp
    stage_index(si, idx, at, L, T, img, l);
    gather_windows<32>(x, img, img < Nimg, si, C, S, T, [&](int k, uint32_t lo, uint32_t hi) { sp[lane * 17 + (k >> 1)] = lo | (hi << 16); });
  };
  auto wval = [&](int m, int k) -> uint32_t { return m < M && k < K ? (uint32_t)__ldg(w + (long long)m * K + k) : 0u; };
  for (int i = threadIdx.x; i < MT * 256; i += blockDim.x) {
    const int r = i & 3, ln = (i >> 2) & 31, ks = (i >> 7) & 1, mt = i >> 8;
    const int m = mt * 16 + (ln >> 2) + 8 * (r & 1), k = ks * 16 + 2 * (ln & 3) + 8 * (r >> 1);
    wf[i] = wval(m, k) | (wval(m, k + 1) << 16);
  }
  for (int i = threadIdx.x; i < MT * 16; i += blockDim.x) sbias[i] = bias != nullptr && i < M ? raw16_to_float(__ldg(bias + i), bf16) : 0.f;
  if (at.img < Nimg) fetch();                              // in flight with the weights
  __syncthreads();
  while (at.img < Nimg) {
    long long run[8 / V];
    run_starts<V>(run, at, t, Nimg, M, L);
    uint32_t b[4][2][2];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t* row = sp + ((g >> 1) * 8 + 2 * j + (g & 1)) * 17 + t;      // position of column n = g
#pragma unroll
      for (int ks = 0; ks < 2; ks++)
#pragma unroll
        for (int r = 0; r < 2; r++) b[j][ks][r] = row[ks * 8 + r * 4];
    }
    const bool live = img < Nimg;
    uint16_t* yl = y + (live ? (long long)img * M * L + l : 0);     // this lane's position, channel 0
    for (int mt = 0; mt < MT; mt++) {
      const float b0 = sbias[mt * 16 + g], b1 = sbias[mt * 16 + g + 8];
      float c[4][4];
      uint32_t af[2][4];
#pragma unroll
      for (int ks = 0; ks < 2; ks++) {
        const uint4 u = *reinterpret_cast<const uint4*>(wf + ((mt * 2 + ks) * 32 + lane) * 4);
        af[ks][0] = u.x; af[ks][1] = u.y; af[ks][2] = u.z; af[ks][3] = u.w;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        c[j][0] = c[j][1] = b0;
        c[j][2] = c[j][3] = b1;
#pragma unroll
        for (int ks = 0; ks < 2; ks++) mma16816(c[j], af[ks], b[j][ks], bf16);
      }
      if (V <= 2) __syncwarp();                            // the windows, or the block before, have been read
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int m = mt * 16 + g + 8 * r;
        if (V > 2 && m >= M) continue;
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = float_to_raw16(c[j][2 * r], bf16) | ((uint32_t)float_to_raw16(c[j][2 * r + 1], bf16) << 16);
        if (V > 2) {
          store8<V>(y + (long long)m * L, v, run);
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) sp[(g + 8 * r) * 17 + 4 * t + j] = v[j];
        }
      }
      if (V <= 2) {
        // planes that no wide run divides: the block of 16 channels turns around in shared memory, so that a store takes 32
        // consecutive positions (64 images of 8 x 28 x 28 to 32 channels, 2 x 2: runs of two bytes 17.4 us, this 8.9)
        __syncwarp();
        const uint16_t* sh = reinterpret_cast<const uint16_t*>(sp) + lane;
        const int rows = min(16, M - mt * 16);
        if (live) {
          uint16_t* d = yl + (long long)mt * 16 * L;
#pragma unroll 4
          for (int r = 0; r < rows; r++) d[(long long)r * L] = sh[r * 34];
        }
      }
    }
    at.advance(by, L);
    if (at.img < Nimg) fetch();
  }
}

// dW[m][k] = sum over positions p (all images) of dy[p][m] * window[p][k]: A = dy (16 channels x 16 positions), B = windows (16
// positions x 8 k).  Slots 2t, 2t + 1 and 2t + 8, 2t + 9 of k-step s are positions 8t + 4s + {0, 1} and {2, 3} of the
// warp's 32, so a lane reads eight consecutive values of a channel.  A warp keeps 64 (or 32) channels x 32 k in
// registers; the CTA's warps are added in order and the CTA writes one partial matrix.  blockIdx.y: group of channels.
template <int MT, int V>
__global__ void __launch_bounds__(kSmallWarps * 32, 2)
conv_wgrad_small_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ dy, const int* __restrict__ idx,
                        float* __restrict__ part, int Nimg, int C, int S, int L, int T, int M, int bf16) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) uint32_t dsm[];
  const int K = C * T, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  int* si = reinterpret_cast<int*>(dsm) + warp * 32 * (T + 17);
  uint16_t* sp = reinterpret_cast<uint16_t*>(si + 32 * T);   // [32 k][32 positions], pitch 34
  const int m0 = blockIdx.y * (MT * 16);
  float acc[MT][4][4];
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;
  SmallPos at((blockIdx.x * kSmallWarps + warp) * 32u, L);
  const SmallPos by(gridDim.x * kSmallWarps * 32u, L);
  for (; at.img < Nimg; at.advance(by, L)) {
    int img;
    unsigned l;
    stage_index(si, idx, at, L, T, img, l);
    long long run[8 / V];
    run_starts<V>(run, at, t, Nimg, M, L);
    gather_windows<MT == 4 ? 8 : 16>(x, img, img < Nimg, si, C, S, T, [&](int k, uint32_t lo, uint32_t hi) {
      sp[k * 34 + lane] = (uint16_t)lo;
      sp[(k + 1) * 34 + lane] = (uint16_t)hi;
    });
    uint32_t b[4][2][2];
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const uint32_t* row = reinterpret_cast<const uint32_t*>(sp) + (nt * 8 + g) * 17 + 4 * t;   // positions 8t ..
#pragma unroll
      for (int h = 0; h < 2; h++)                        // k-steps
#pragma unroll
        for (int r = 0; r < 2; r++) b[nt][h][r] = row[2 * h + r];
    }
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
      uint32_t lo[4], hi[4];
      load8<V>(dy + (long long)(m0 + mt * 16 + g) * L, lo, run);
      load8<V>(dy + (long long)(m0 + mt * 16 + g + 8) * L, hi, run);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t af[4] = {lo[2 * h], hi[2 * h], lo[2 * h + 1], hi[2 * h + 1]};
#pragma unroll
        for (int nt = 0; nt < 4; nt++) mma16816(acc[mt][nt], af, b[nt][h], bf16);
      }
    }
  }
  __syncthreads();
  float* red = reinterpret_cast<float*>(dsm);            // [MT * 16][32], reusing the index rows
  for (int w = 0; w < kSmallWarps; w++) {
    if (warp == w) {
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int nt = 0; nt < 4; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            float* d = red + (mt * 16 + g + 8 * (e >> 1)) * kDirectK + nt * 8 + 2 * t + (e & 1);
            *d = w == 0 ? acc[mt][nt][e] : *d + acc[mt][nt][e];
          }
    }
    __syncthreads();
  }
  float* out = part + ((long long)blockIdx.x * M + m0) * K;
  for (int i = threadIdx.x; i < MT * 16 * K; i += blockDim.x) out[i] = red[(i / K) * kDirectK + i % K];
}

// Widest run of positions that stays aligned from image to image.
inline int run_width(int L, const void* p) {
  const uintptr_t a = (uintptr_t)p;
  if (L % 8 == 0 && (a & 15) == 0) return 8;
  if (L % 4 == 0 && (a & 7) == 0) return 4;
  if (L % 2 == 0 && (a & 3) == 0) return 2;
  return 1;
}

inline int wgrad_small_ctas(long long P) {
  long long g = (P + 255) / 256;
  if (g > 2 * 148) g = 2 * 148;
  return g < 1 ? 1 : (int)g;
}
inline bool wgrad_small_ok(int C, int T, int M) { return C * T <= kDirectK && (M == 32 || M == 64 || M == 128); }

int set_attr_once() {
  static bool done = false;
  if (!done) {
    GB_CUDA_OK(cudaFuncSetAttribute(conv_igemm_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, CSMEM));
    GB_CUDA_OK(cudaFuncSetAttribute(conv_igemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, CSMEM));
    done = true;
  }
  return gbh::E_OK;
}

}  // namespace

int gbc::launch_wgrad_finish(const float* part, uint16_t* dW, int M, int C, int T, int splits, int bf16, int beta, bool tap_major,
                             cudaStream_t s) {
  const long long n = (long long)M * C * T, blocks = (n + 31) / 32;
  gbh::launch(conv_wgrad_finish_kernel, dim3((int)(blocks < 148 * 16 ? blocks : 148 * 16)), dim3(256), 0, s, 1, part, dW, n, C, T, splits, bf16, beta, tap_major);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

enum { DT_BF16 = 0, DT_F16 = 1 };

// y[n][m][l] = bias[m] + sum_{c,tap} W[m][c * T + tap] * x[n][c][idx[l][tap]] for 16-bit tensors.
// w: (M, C * T) row-major.  The forward passes the (C_out, C_in, T) weights as they are; the data
// gradient passes x := dy, idx := the inverse map and the weights regrouped as (C_in, C_out * T).
// ktab: gb_conv_ktab_len(C, T) int pairs {c * S, tap} ({-1, 0} past C * T), built once per geometry.
GB_EXPORT int gb_conv_ktab_len(int C, int T) { return (C * T + 127) / 128 * 128; }

GB_EXPORT int gb_conv_igemm(int dtype, const void* x, const void* w, const int* ktab, const int* idx,
                            const void* bias, void* y, int Nimg, int C, int S, int L, int T, int M, void* stream) {
  if (dtype != DT_BF16 && dtype != DT_F16) {
    gbh::set_error("gb_conv_igemm: bf16 or fp16 tensors");
    return gbh::E_BAD_ARG;
  }
  if (Nimg <= 0 || C <= 0 || L <= 0 || T <= 0 || M <= 0 || Nimg > 65535 || T > CMAX_T_SMEM ||
      (long long)C * S >= (1LL << 31) || (long long)M * L >= (1LL << 31) || (long long)Nimg * L >= (1LL << 31) - CBN) {
    gbh::set_error("gb_conv_igemm: geometry out of range (at most %d taps, 65535 images)", CMAX_T_SMEM);
    return gbh::E_BAD_ARG;
  }
  int rc = set_attr_once();
  if (rc) return rc;
  ConvArgs a;
  memset(&a, 0, sizeof(a));
  a.W = (const uint16_t*)w;
  a.w_vec = ((C * T) % 8 == 0) && (((uintptr_t)w & 15) == 0);
  a.ktab = (const int2*)ktab;
  a.X = (const uint16_t*)x; a.idx = idx; a.Y = y; a.bias = (const uint16_t*)bias;
  a.Nimg = Nimg; a.C = C; a.S = S; a.L = L; a.T = T; a.M = M;
  a.bf16 = dtype == DT_BF16;
  a.status = gbh::status_ptr();
  dim3 grid((unsigned)(((long long)Nimg * L + CBN - 1) / CBN), (M + CBM - 1) / CBM, 1);
  conv_igemm_kernel<0><<<grid, CTHREADS, CSMEM, (cudaStream_t)stream>>>(a);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// Whether gb_conv_direct_small takes a forward convolution: a contraction of at most 32 and a channel count that is a
// multiple of 4 and at most 372 (the weights of 372 channels in fragment order, 26 KB, and the windows of eight warps, 50 KB
// at 32 taps, fit its limit; more channels fill the 128-wide tiles of the other kernels).
GB_EXPORT int gb_conv_direct_ok(int C, int T, int M) {
  return C * T <= kDirectK && (M & 3) == 0 && M > 0 && M <= 372;
}

// The forward of gb_conv_igemm for the shapes gb_conv_direct_ok accepts (same arguments, no ktab).
GB_EXPORT int gb_conv_direct_small(int dtype, const void* x, const void* w, const int* idx, const void* bias,
                                   void* y, int Nimg, int C, int S, int L, int T, int M, void* stream) {
  if (dtype != DT_BF16 && dtype != DT_F16) {
    gbh::set_error("gb_conv_direct_small: bf16 or fp16 tensors");
    return gbh::E_BAD_ARG;
  }
  if (!gb_conv_direct_ok(C, T, M) || Nimg <= 0 || Nimg > 65535 || L <= 0) {
    gbh::set_error("gb_conv_direct_small: needs C * T <= %d, a channel count that is a multiple of 4, at most 65535 images", kDirectK);
    return gbh::E_BAD_ARG;
  }
  const int mt = (M + 15) / 16;
  const size_t smem = (size_t)mt * 256 * 4 + mt * 16 * 4 + (size_t)kSmallWarps * 32 * (T + 17) * 4;
  const long long blocks = ((long long)Nimg * L + 32 * kSmallWarps - 1) / (32 * kSmallWarps);
  const int grid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
#define GB_DS(V)                                                                                                          \
  {                                                                                                                       \
    GB_CUDA_OK(cudaFuncSetAttribute(conv_direct_small_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem)); \
    gbh::launch(conv_direct_small_kernel<V>, dim3(grid), dim3(kSmallWarps * 32), smem, (cudaStream_t)stream, 1,                                   \
        (const uint16_t*)x, (const uint16_t*)w, idx, (const uint16_t*)bias, (uint16_t*)y, Nimg, C, S, L, T, M, dtype == DT_BF16); \
  }
  switch (run_width(L, y)) {
    case 8: GB_DS(8) break;
    case 4: GB_DS(4) break;
    case 2: GB_DS(2) break;
    default: GB_DS(1)
  }
#undef GB_DS
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// Number of K splits the weight gradient uses for a problem (partials: splits * M * C * T floats).
GB_EXPORT int gb_conv_wgrad_splits(int Nimg, int L, int M, int C, int T) {
  const long long R = (long long)Nimg * L;
  if (wgrad_small_ok(C, T, M)) return wgrad_small_ctas(R);      // one partial matrix per CTA of the direct kernel
  const long long tiles = (long long)((M + CBM - 1) / CBM) * ((C * T + CBN - 1) / CBN);
  long long want = (2 * 148 + tiles - 1) / tiles;          // about two waves of CTAs
  const long long max_splits = (R + 4 * CBK - 1) / (4 * CBK);  // at least four k-blocks per split
  if (want > max_splits) want = max_splits;
  if (want < 1) want = 1;
  if (want > 1024) want = 1024;
  return (int)want;
}

// dW[m][(c,tap)] (+)= sum_{n,l} dy[n][m][l] * x[n][c][idx[l][tap]].  part: gb_conv_wgrad_splits() * M * C * T floats.
GB_EXPORT int gb_conv_wgrad(int dtype, const void* x, const void* dy, const int* ktab, const int* idx, void* dw,
                            float* part, int Nimg, int C, int S, int L, int T, int M, int beta, void* stream) {
  if (dtype != DT_BF16 && dtype != DT_F16) {
    gbh::set_error("gb_conv_wgrad: bf16 or fp16 tensors");
    return gbh::E_BAD_ARG;
  }
  if (T > CMAX_T_SMEM || (long long)C * S >= (1LL << 31) || (long long)M * L >= (1LL << 31)) {
    gbh::set_error("gb_conv_wgrad: geometry out of range");
    return gbh::E_BAD_ARG;
  }
  int rc = set_attr_once();
  if (rc) return rc;
  const int splits = gb_conv_wgrad_splits(Nimg, L, M, C, T);
  const long long R = (long long)Nimg * L;
  if (wgrad_small_ok(C, T, M)) {
    const int bf = dtype == DT_BF16;
    const size_t idx_bytes = (size_t)kSmallWarps * 32 * (T + 17) * 4;
#define GB_WS(MT, V)                                                                                               \
  {                                                                                                                \
    const size_t red = (size_t)MT * 16 * kDirectK * 4, smem = idx_bytes > red ? idx_bytes : red;                   \
    GB_CUDA_OK(cudaFuncSetAttribute(conv_wgrad_small_kernel<MT, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem)); \
    gbh::launch(conv_wgrad_small_kernel<MT, V>, dim3(dim3(splits, M / (MT * 16))), dim3(kSmallWarps * 32), smem, (cudaStream_t)stream, 1,  \
        (const uint16_t*)x, (const uint16_t*)dy, idx, part, Nimg, C, S, L, T, M, bf);                              \
  }
#define GB_WV(MT)                    \
  switch (run_width(L, dy)) {        \
    case 8: GB_WS(MT, 8) break;      \
    case 4: GB_WS(MT, 4) break;      \
    case 2: GB_WS(MT, 2) break;      \
    default: GB_WS(MT, 1)            \
  }
    if (M == 32) { GB_WV(2) } else { GB_WV(4) }
#undef GB_WV
#undef GB_WS
    return gbc::launch_wgrad_finish(part, (uint16_t*)dw, M, C, T, splits, bf, beta, false, (cudaStream_t)stream);
  }
  long long per = (R + splits - 1) / splits;
  per = (per + CBK - 1) / CBK * CBK;
  ConvArgs a;
  memset(&a, 0, sizeof(a));
  a.X = (const uint16_t*)x; a.DY = (const uint16_t*)dy; a.idx = idx; a.Y = part;
  a.ktab = (const int2*)ktab;
  a.Nimg = Nimg; a.C = C; a.S = S; a.L = L; a.T = T; a.M = M;
  a.bf16 = dtype == DT_BF16;
  a.r_per_split = per;
  a.status = gbh::status_ptr();
  const int K = C * T;
  dim3 grid((K + CBN - 1) / CBN, (M + CBM - 1) / CBM, splits);
  conv_igemm_kernel<1><<<grid, CTHREADS, CSMEM, (cudaStream_t)stream>>>(a);
  return gbc::launch_wgrad_finish(part, (uint16_t*)dw, M, C, T, splits, a.bf16, beta, false, (cudaStream_t)stream);
}
