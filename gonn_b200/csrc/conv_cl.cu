// Implicit-GEMM convolution over channels-last copies: forward, data gradient and weight gradient for
// 16-bit tensors whose contracted channel counts are multiples of 8.
//
// conv.cu gathers its operands element by element: 64 two-byte loads, index look-ups and selects per row and
// 64-wide k-block bound it (140 us for 43 264 positions x 576 x 128, 4 us of tensor-core time).  Here one pass turns
// the (N, C, S) tensors into (N, S, C) (both fit L2; 8 us for 7 MB of images), so that eight channels of a window tap are one
// 16-byte cp.async with zero fill for the padding, and the contraction runs over (tap, channel):
//   forward   y[n][m][l]   = bias[m] + sum_{tap,c} Wp[m][tap][c] * xt[n][idx[l][tap]][c]
//   dgrad     the same with xt := dy channels-last, idx := the inverse map, Wp := (C_in, tap, C_out)
//   wgrad     dWp[m][(tap,c)] = sum_{p = (n, l)} dyt[p][m] * xt[n][idx[l][tap]][c], split over CTAs along p; both
//             operands are staged as rows of positions (MN-major), the form tcgen05 reads without a transpose
// Tiles 128 x 128 x 64, 32 KB stages: eight producer warps issue the copies of one stage while the
// previous one lands, one elected thread issues the MMAs.  Measured at 256 images, 64 -> 128
// channels, 3 x 3 on 15 x 15: forward 31 us (140), dgrad 50 (141), wgrad 39 (110), packing included.
//
// No tensor map and no cluster is involved.  Every wait is bounded.
#include "conv.cuh"

using namespace gb;

namespace {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int TILE = 128 * BK * 2, STAGE = 2 * TILE;
constexpr int PRODUCERS = 256, THREADS = PRODUCERS + 32;
constexpr int MAX_T = 32;
// Three stages, two in flight, two CTAs per SM.  All three in flight make the next copy wait for the MMAs of the
// block that has just landed (forward 31 -> 42 us); one CTA with six stages has too few warps issuing (wgrad 39 -> 60).
constexpr int STAGES = 3, LAG = 1;
constexpr int smem_bytes(int T) { return STAGES * STAGE + 1024 /*alignment*/ + 256 /*barriers*/ + BN * T * 4; }

struct ClArgs {
  const uint16_t* W;       // forward / dgrad: (M, T * C), k = tap * C + c
  const uint16_t* X;       // (Nimg * S, C)
  const uint16_t* DY;      // wgrad: (Nimg * L, M)
  const int* idx;          // [L][T]
  void* Y;                 // forward / dgrad: (Nimg, M, L); wgrad: fp32 partials [splits][M][T * C]
  const uint16_t* bias;
  int Nimg, C, S, L, T, M;
  int bf16;
  long long per_split;     // wgrad: positions per split (a multiple of 64)
  int* status;
};

// MODE 0: forward / dgrad (grid: position tiles, M tiles); MODE 1: wgrad (grid: (tap, c) tiles, M tiles, splits)
template <int MODE>
__global__ void __launch_bounds__(THREADS, 2) conv_cl_kernel(const ClArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE);
  uint64_t* full_bar = bars;               // [STAGES], one arrival per producer warp
  uint64_t* empty_bar = bars + STAGES;     // [STAGES], tcgen05.commit
  uint64_t* done_bar = bars + 2 * STAGES;
  uint32_t* tmem_slot = (uint32_t*)(done_bar + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  int* sidx = reinterpret_cast<int*>(smem + STAGES * STAGE + 256);   // MODE 0: [T][128] source rows of the tile's positions
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = a.C * a.T;
  const long long P = (long long)a.Nimg * a.L;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(&full_bar[s], PRODUCERS / 32); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  pdl_wait();
  const int m0 = blockIdx.y * BM;
  const long long n0 = (long long)blockIdx.x * BN;        // MODE 0: position; MODE 1: (tap, c) column
  if (MODE == 0) {
    for (int i = threadIdx.x; i < BN * a.T; i += THREADS) {
      const int tap = i >> 7;
      const long long p = n0 + (i & 127);
      int src = -1;
      if (p < P) {
        const unsigned img = (unsigned)p / (unsigned)a.L, l = (unsigned)p - img * (unsigned)a.L;   // P < 2^31
        src = __ldg(a.idx + (long long)l * a.T + tap);
        if (src >= 0) src += (int)img * a.S;
      }
      sidx[i] = src;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  long long k_begin = 0, k_end = K;                       // contraction range: k (MODE 0) or positions (MODE 1)
  if (MODE == 1) {
    k_begin = (long long)blockIdx.z * a.per_split;
    k_end = min(k_begin + a.per_split, P);
  }
  const int nkb = k_end > k_begin ? (int)((k_end - k_begin + BK - 1) / BK) : 0;

  if (warp < 8) {
    const int c8 = threadIdx.x & 7, r0 = threadIdx.x >> 3;      // 16-byte piece of a row, rows r0 + 32 i
    const uint32_t ring = smem_u32(smem);
    bool ok = true;
    int stage = 0;
    uint32_t phase = 0;
    // MODE 0: this thread's k of the current k-block as (tap, c)
    int tap = 0, c = c8 * 8;
    // MODE 1: columns h * 64 + c8 * 8 of the tile as (tap, c), the two positions of this thread and their index entries
    int tap_h[2] = {0, 0}, c_h[2] = {0, 0}, img[2], l[2], src[2][2];
    bool n_ok[2] = {false, false};
    if (MODE == 0) {
      while (c >= a.C) { c -= a.C; tap++; }
    } else {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int n = (int)n0 + h * 64 + c8 * 8;
        n_ok[h] = n < K;
        tap_h[h] = n_ok[h] ? n / a.C : 0;
        c_h[h] = n - tap_h[h] * a.C;
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const long long p = k_begin + r0 + 32 * i;
        img[i] = (int)(p / a.L);
        l[i] = (int)(p - (long long)img[i] * a.L);
      }
    }
    auto fetch_src = [&](int kb) {                         // MODE 1: index entries of k-block kb (l, img stand there)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const bool live = k_begin + (long long)kb * BK + r0 + 32 * i < k_end;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          src[i][h] = live && n_ok[h] ? __ldg(a.idx + (long long)l[i] * a.T + tap_h[h]) : -1;
          if (src[i][h] >= 0) src[i][h] += img[i] * a.S;
        }
        l[i] += BK;
        while (l[i] >= a.L) { l[i] -= a.L; img[i]++; }
      }
    };
    if (MODE == 1 && nkb > 0) fetch_src(0);
    for (int kb = 0; kb < nkb; kb++) {
      if (lane == 0) ok = mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, a.status, ST_CONV_TIMEOUT, 1);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      const uint32_t sa = ring + stage * STAGE, sb = sa + TILE;
      if (MODE == 0) {
        const int k = kb * BK + c8 * 8;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = r0 + 32 * i;
          const uint32_t off = r * 128 + ((c8 ^ (r & 7)) << 4);
          if (m0 + 32 * i < a.M) {                         // rows of the accumulator past M are never read
            const bool live = m0 + r < a.M && k < K;
            cp_async16(sa + off, a.W + (live ? (long long)(m0 + r) * K + k : 0), live ? 16 : 0);
          }
          const int s = tap < a.T ? sidx[tap * BN + r] : -1;
          cp_async16(sb + off, a.X + (s >= 0 ? (long long)s * a.C + c : 0), s >= 0 ? 16 : 0);
        }
        c += BK;
        while (c >= a.C) { c -= a.C; tap++; }
      } else {
        const long long p0 = k_begin + (long long)kb * BK;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int r = r0 + 32 * i;
          const uint32_t off = r * 128 + ((c8 ^ (r & 7)) << 4);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int m = m0 + h * 64 + c8 * 8;
            if (m0 + h * 64 < a.M) {
              const bool live = m < a.M && p0 + r < k_end;
              cp_async16(sa + h * (TILE / 2) + off, a.DY + (live ? (p0 + r) * a.M + m : 0), live ? 16 : 0);
            }
            cp_async16(sb + h * (TILE / 2) + off, a.X + (src[i][h] >= 0 ? (long long)src[i][h] * a.C + c_h[h] : 0), src[i][h] >= 0 ? 16 : 0);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (MODE == 1 && kb + 1 < nkb) fetch_src(kb + 1);
      if (kb >= LAG) {                                     // k-block kb - LAG has landed
        asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[(kb - LAG) % STAGES]);
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_proxy_async_smem();
    __syncwarp();
    if (ok && lane == 0)
      for (int kb = nkb > LAG ? nkb - LAG : 0; kb < nkb; kb++) mbar_arrive(&full_bar[kb % STAGES]);
  } else if (elect_one()) {
    uint32_t id = make_idesc(1u, 0u, MODE == 1, MODE == 1, BM, BN);
    if (a.bf16) id |= (1u << 7) | (1u << 10);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < nkb; kb++) {
      if (!mbar_wait(&full_bar[stage], phase, abort_flag, a.status, ST_CONV_TIMEOUT, 2)) break;
      tc_fence_after();
      const uint32_t sa = smem_u32(smem + stage * STAGE), sb = sa + TILE;
#pragma unroll
      for (int k = 0; k < BK / 16; k++) {
        // MODE 0, K-major: 8-row groups 1024 B apart, a step is 32 B along K.  MODE 1, MN-major: the two 64-column
        // blocks TILE / 2 apart, 8-row k groups 1024 B apart, a step is 16 rows.
        const uint64_t da = MODE == 0 ? make_smem_desc_sw128(sa + k * 32, 16, 1024) : make_smem_desc_sw128(sa + k * 2048, TILE / 2, 1024);
        const uint64_t db = MODE == 0 ? make_smem_desc_sw128(sb + k * 32, 16, 1024) : make_smem_desc_sw128(sb + k * 2048, TILE / 2, 1024);
        tc_mma_f16(tmem_base, da, db, id, kb > 0 || k != 0);
      }
      tc_commit(&empty_bar[stage]);
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    tc_commit(done_bar);
  }

  // ---- epilogue: a warp's 32 x 32 blocks turn around in shared memory (the ring is idle), lanes run along the columns ----
  if (warp < 8) {
    bool ok = true;
    if (lane == 0) ok = mbar_wait(done_bar, 0, abort_flag, a.status, ST_CONV_TIMEOUT, 3);
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    const int q = warp & 3, half = warp >> 2;              // TMEM lane quarter, column half
    const int mrow0 = m0 + q * 32;
    if (ok && mrow0 < a.M) {
      tc_fence_after();
      float* stf = reinterpret_cast<float*>(smem + warp * (32 * 33 * 4));
      const int rows = min(32, a.M - mrow0);
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
        const float bv = MODE == 0 && a.bias != nullptr && lane < rows ? gbc::raw16_to_float(__ldg(a.bias + mrow0 + lane), a.bf16) : 0.f;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; j++) stf[lane * 33 + j] = __uint_as_float(r[j]) + bv;
        __syncwarp();
        const long long n = n0 + col0 + lane;
        if (MODE == 0) {
          if (n < P) {
            const unsigned img = (unsigned)n / (unsigned)a.L, l = (unsigned)n - img * (unsigned)a.L;
            uint16_t* yb = (uint16_t*)a.Y + ((long long)img * a.M + mrow0) * a.L + l;
#pragma unroll 8
            for (int rr = 0; rr < rows; rr++) yb[(long long)rr * a.L] = gbc::float_to_raw16(stf[rr * 33 + lane], a.bf16);
          }
        } else if (n < K) {
          float* pb = (float*)a.Y + ((long long)blockIdx.z * a.M + mrow0) * K + n;
#pragma unroll 8
          for (int rr = 0; rr < rows; rr++) pb[(long long)rr * K] = stf[rr * 33 + lane];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem_base, BN);
}

// One job turns (n, rows, cols) into (n, cols, rows): images to channels-last, or weights to (tap, channel) order.
struct PackJob {
  const uint16_t* src;
  uint16_t* dst;
  int n, rows, cols;
  int tr, tc;              // tiles of 64 along rows and cols
  long long first;         // index of the job's first block
  long long s_n, s_r, s_c; // source strides: a weight is read as (C_in, C_out, tap) without a copy
};
struct PackArgs {
  PackJob job[3];
  int jobs;
};

// A block of 256 threads turns a 64 x 64 tile.  Two-byte loads along the contiguous dimension, pairs of rows
// packed into one word of shared memory (pitch 33 words: free of conflicts both ways), 16-byte stores.
__global__ void __launch_bounds__(256) conv_pack_kernel(const PackArgs a) {
  pdl_trigger();
  pdl_wait();
  __shared__ uint32_t sm[64 * 33];
  int ji = 0;
  while (ji + 1 < a.jobs && (long long)blockIdx.x >= a.job[ji + 1].first) ji++;
  const PackJob& j = a.job[ji];
  long long t = (long long)blockIdx.x - j.first;
  const int ct = (int)(t % j.tc);
  t /= j.tc;
  const int rt = (int)(t % j.tr), n = (int)(t / j.tr);
  const uint16_t* src = j.src + n * j.s_n;
  const int c = threadIdx.x & 63;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int r = 2 * ((threadIdx.x >> 6) + 4 * i);
    const int gr = rt * 64 + r, gc = ct * 64 + c;
    uint32_t v = 0;
    if (gc < j.cols) {
      const uint16_t* p = src + gr * j.s_r + gc * j.s_c;
      if (gr < j.rows) v = __ldg(p);
      if (gr + 1 < j.rows) v |= (uint32_t)__ldg(p + j.s_r) << 16;
    }
    sm[c * 33 + (r >> 1)] = v;
  }
  __syncthreads();
  uint16_t* dst = j.dst + (long long)n * j.rows * j.cols;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int q = threadIdx.x + 256 * i, col = q >> 3, c8 = q & 7;
    const int gc = ct * 64 + col, gr = rt * 64 + c8 * 8;
    if (gc >= j.cols || gr >= j.rows) continue;
    const uint32_t* s = sm + col * 33 + c8 * 4;
    *reinterpret_cast<uint4*>(dst + (long long)gc * j.rows + gr) = make_uint4(s[0], s[1], s[2], s[3]);   // rows % 8 == 0
  }
}

int add_job(PackArgs& pa, long long& blocks, const void* src, void* dst, int n, int rows, int cols, long long s_n, long long s_r,
            long long s_c) {
  PackJob& j = pa.job[pa.jobs++];
  j.src = (const uint16_t*)src; j.dst = (uint16_t*)dst;
  j.n = n; j.rows = rows; j.cols = cols;
  j.tr = (rows + 63) / 64; j.tc = (cols + 63) / 64;
  j.s_n = s_n; j.s_r = s_r; j.s_c = s_c;
  j.first = blocks;
  blocks += (long long)n * j.tr * j.tc;
  return 0;
}

int configure() {
  GB_CUDA_OK(cudaFuncSetAttribute(conv_cl_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MAX_T)));
  GB_CUDA_OK(cudaFuncSetAttribute(conv_cl_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(0)));
  return gbh::E_OK;
}

// positions per split of the weight gradient: one CTA per SM and at least four k-blocks each
int wgrad_splits(long long P, int M, int K) {
  const long long tiles = (long long)((M + BM - 1) / BM) * ((K + BN - 1) / BN);
  long long want = 148 / tiles;
  const long long most = (P + 4 * BK - 1) / (4 * BK);
  if (want > most) want = most;
  return want < 1 ? 1 : (int)want;
}

bool geometry_ok(int Nimg, int C, int S, int L, int T, int M) {
  return Nimg > 0 && C > 0 && S > 0 && L > 0 && T > 0 && M > 0 && T <= MAX_T && (long long)C * T < (1LL << 31) &&
         (long long)Nimg * S < (1LL << 31) && (long long)Nimg * L < (1LL << 31) - BN && (long long)C * S < (1LL << 31) &&
         (long long)M * L < (1LL << 31);
}

}  // namespace

// 16-bit elements of the scratch that gb_conv_cl_fwd / gb_conv_cl_bwd need (a 16-byte aligned buffer).
GB_EXPORT long long gb_conv_cl_fwd_ws(int Nimg, int C, int S, int T, int M) {
  return (long long)Nimg * S * C + (long long)M * T * C;
}
GB_EXPORT long long gb_conv_cl_bwd_ws(int Nimg, int C, int S, int L, int T, int M, int need_dx, int need_dw) {
  return (long long)Nimg * L * M + (need_dw ? (long long)Nimg * S * C : 0) + (need_dx ? (long long)M * T * C : 0);
}
// fp32 elements of the weight gradient's partial sums.
GB_EXPORT long long gb_conv_cl_part(int Nimg, int C, int L, int T, int M) {
  return (long long)wgrad_splits((long long)Nimg * L, M, C * T) * M * C * T;
}
// 1 when the channels-last kernels take the geometry (multiples of 8 contracted channels: C_in forward, both backward).  A
// forward of one tap reads every element once: the gathers of conv.cu beat a pass that packs first (8 images of 256 x 56 x 56
// to 64 channels: 49 | 57 us; backward 150 | 131; 3 x 3 from 64 to 64 there: 157 | 84 and 410 | 211).
GB_EXPORT int gb_conv_cl_ok(int Nimg, int C, int S, int L, int T, int M, int bwd) {
  return C % 8 == 0 && (bwd ? M % 8 == 0 : T > 1) && geometry_ok(Nimg, C, S, L, T, M) ? 1 : 0;
}

// y (Nimg, M, L) = bias + W * windows of x; x (Nimg, C, S), w (M, C, T), idx [L][T].
GB_EXPORT int gb_conv_cl_fwd(int dtype, const void* x, const void* w, const int* idx, const void* bias, void* y, void* ws,
                             int Nimg, int C, int S, int L, int T, int M, void* stream) {
  if (dtype > 1 || dtype < 0 || !gb_conv_cl_ok(Nimg, C, S, L, T, M, 0) || ((uintptr_t)ws & 15)) {
    gbh::set_error("gb_conv_cl_fwd: 16-bit tensors, C a multiple of 8, at most %d taps", MAX_T);
    return gbh::E_BAD_ARG;
  }
  int rc = configure();
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  uint16_t* xt = (uint16_t*)ws;
  uint16_t* wp = xt + (long long)Nimg * S * C;
  PackArgs pa;
  memset(&pa, 0, sizeof(pa));
  long long blocks = 0;
  add_job(pa, blocks, x, xt, Nimg, C, S, (long long)C * S, S, 1);
  add_job(pa, blocks, w, wp, M, C, T, (long long)C * T, T, 1);
  if (blocks >= (1LL << 31)) {
    gbh::set_error("gb_conv_cl_fwd: problem too large");
    return gbh::E_TOO_LARGE;
  }
  gbh::launch(conv_pack_kernel, dim3((unsigned)blocks), dim3(256), 0, s, 1, pa);
  ClArgs a;
  memset(&a, 0, sizeof(a));
  a.W = wp; a.X = xt; a.idx = idx; a.Y = y; a.bias = (const uint16_t*)bias;
  a.Nimg = Nimg; a.C = C; a.S = S; a.L = L; a.T = T; a.M = M; a.bf16 = dtype == 0;
  a.status = gbh::status_ptr();
  gbh::launch(conv_cl_kernel<0>, dim3(dim3((unsigned)(((long long)Nimg * L + BN - 1) / BN), (M + BM - 1) / BM)), dim3(THREADS), smem_bytes(T), s, 1, a);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// dx (Nimg, C, S) when not null, through the inverse map inv [S][T]; dw (M, C, T) (+ dw when beta) when not null.
GB_EXPORT int gb_conv_cl_bwd(int dtype, const void* x, const void* w, const void* dy, const int* idx, const int* inv, void* dx,
                             void* dw, int beta, void* ws, float* part, int Nimg, int C, int S, int L, int T, int M, void* stream) {
  if (dtype > 1 || dtype < 0 || !gb_conv_cl_ok(Nimg, C, S, L, T, M, 1) || ((uintptr_t)ws & 15)) {
    gbh::set_error("gb_conv_cl_bwd: 16-bit tensors, channel counts that are multiples of 8, at most %d taps", MAX_T);
    return gbh::E_BAD_ARG;
  }
  int rc = configure();
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  uint16_t* dyt = (uint16_t*)ws;
  uint16_t* next = dyt + (long long)Nimg * L * M;
  uint16_t *xt = nullptr, *wp = nullptr;
  PackArgs pa;
  memset(&pa, 0, sizeof(pa));
  long long blocks = 0;
  add_job(pa, blocks, dy, dyt, Nimg, M, L, (long long)M * L, L, 1);
  if (dw != nullptr) {
    xt = next;
    next += (long long)Nimg * S * C;
    add_job(pa, blocks, x, xt, Nimg, C, S, (long long)C * S, S, 1);
  }
  if (dx != nullptr) {
    wp = next;                                             // (C, T, M): for each input channel, rows = M, cols = T
    add_job(pa, blocks, w, wp, C, M, T, T, (long long)C * T, 1);
  }
  if (blocks >= (1LL << 31)) {
    gbh::set_error("gb_conv_cl_bwd: problem too large");
    return gbh::E_TOO_LARGE;
  }
  gbh::launch(conv_pack_kernel, dim3((unsigned)blocks), dim3(256), 0, s, 1, pa);
  ClArgs a;
  memset(&a, 0, sizeof(a));
  a.bf16 = dtype == 0; a.Nimg = Nimg; a.T = T; a.status = gbh::status_ptr();
  if (dx != nullptr) {
    a.W = wp; a.X = dyt; a.idx = inv; a.Y = dx;
    a.C = M; a.S = L; a.L = S; a.M = C;
    gbh::launch(conv_cl_kernel<0>, dim3(dim3((unsigned)(((long long)Nimg * S + BN - 1) / BN), (C + BM - 1) / BM)), dim3(THREADS), smem_bytes(T), s, 1, a);
  }
  if (dw != nullptr) {
    const long long P = (long long)Nimg * L;
    const int splits = wgrad_splits(P, M, C * T);
    a.W = nullptr; a.X = xt; a.DY = dyt; a.idx = idx; a.Y = part;
    a.C = C; a.S = S; a.L = L; a.M = M;
    a.per_split = ((P + splits - 1) / splits + BK - 1) / BK * BK;
    gbh::launch(conv_cl_kernel<1>, dim3(dim3((C * T + BN - 1) / BN, (M + BM - 1) / BM, splits)), dim3(THREADS), smem_bytes(0), s, 1, a);
    rc = gbc::launch_wgrad_finish(part, (uint16_t*)dw, M, C, T, splits, a.bf16, beta, true, s);
    if (rc) return rc;
  }
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}
