// Flash attention for sm_100a: forward and backward on tcgen05 tensor cores
// with the score tile, the probability tile and the output accumulator in
// tensor memory.
//
// Math follows the reference's fused kernels (backend/cuda/gonn_cuda.cu:302-450
// forward with online softmax and L = m + log(l); :333-383 backward identities
// p = exp(s*scale - L), D = dO.O, dV += p^T dO, dS = p (dO.v - D) scale,
// dQ += dS k, dK += dS^T q) and the scale 1/sqrt(d) and causal rule k <= q of
// nn/attention.go:124-147.  The design is new: 128-row tiles, bf16/fp16 operands,
// fp32 accumulation, no atomics (dQ and dK/dV are produced by two kernels so that
// every output tile has one owner and a fixed summation order).
//
// Forward CTA (192 threads, two or four CTAs per SM) owns 128 query rows of one (batch, head):
//   warp 0      TMA loads of Q once and the K / V sub-tiles of 64 keys (rings)
//   warp 1      MMA issue: S = Q K^T into one of two TMEM score buffers, then
//               O += P V with P read from TMEM (written there by the softmax warps)
//   warps 2-5   softmax: one thread per row; running max / sum in registers;
//               O is rescaled only when the max moved by more than 2^8
// Backward: a row-statistics kernel (Delta = dO . O), then one CTA per 128-key tile for
// dK / dV, which leaves dS^T behind for one product dQ = dS K (or, without room for it, one CTA per 128-query tile that
// computes the scores again); both stream 64-row sub-tiles and keep S and dP in TMEM.
// Tensors are addressed through 4-D tensor maps (d, s, h, b) with arbitrary
// strides, so (B,S,H,D) and (B,H,S,D) layouts both work without copies.
#include "common.cuh"

#include <type_traits>

using namespace gb;

namespace {

constexpr int BQ = 128;   // query rows per tile
constexpr int BKV = 128;  // key rows per tile
constexpr int kFwdThreads = 192;

struct AttnArgs {
  int B, H, Sq, Sk;
  int D;  // the tensors' head size: a multiple of 8, at most the kernel's HD (TMA zero-fills the rest)
  float scale_log2;  // scale * log2(e)
  float scale;
  int causal;
  int in_bf16;
  float* LSE;  // [B, H, Sq]
  // backward
  const float* Delta;  // [B, H, Sq]
  void* dQ;
  long long dq_sb, dq_ss, dq_sh;  // element strides (b, s, h); d is contiguous
  // optional spill of dS^T from the dK/dV kernel: [B*H][ds_rows keys][ds_ld queries], 16-bit, already
  // multiplied by the softmax scale.  When set, dQ is one product of this matrix with K
  // (fa_bwd_dq_ds_kernel) instead of a second pass that recomputes S, P and dP.
  void* dS;
  long long ds_ld, ds_rows;
  int* status;
  // optional timeline of CTA (0,0,0) of the dK/dV kernel: [3 lanes][kTraceSlots] SM clock stamps
  long long* trace;
  float inv_scale;       // of the scale that the row statistics are folded with (see stat_row)
  int head_group;        // causal launch order, see block_of(); reciprocals, rounded up, times 2^32, of it and of H
  unsigned group_recip, head_recip;
};

// The tile (by rank: longest first) and head of this CTA.  Causal tiles differ in length by the number of tiles.  In the
// grid's own order a head's tiles run together, longest first, and the last head's longest tile starts when everything
// else has ended; the last `head_group` heads therefore start their longest tiles first, then their second longest, and
// so on, and the kernel ends on the shortest.  (Interleaving more heads than that loses their operands' and the
// spilled dS's locality in L2.)  Quotients are products with reciprocals.
__device__ __forceinline__ void block_of(const AttnArgs& args, int& rank, int& h, int& b) {
  rank = blockIdx.x;
  h = blockIdx.y;
  b = blockIdx.z;
  const unsigned first = gridDim.y * gridDim.z - args.head_group;
  const unsigned lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (args.head_group > 0 && lin >= first * gridDim.x) {
    const unsigned in = lin - first * gridDim.x, r = __umulhi(in, args.group_recip), bh = first + in - r * args.head_group;
    rank = r;
    b = __umulhi(bh, args.head_recip);
    h = bh - b * gridDim.y;
  }
}

constexpr int kTraceSlots = 512;
// lane: 0 = MMA thread, 1 / 2 = first warp of elementwise group 0 / 1
// Compiled in only with -DGB_FA_TRACE: a stamp costs its warp registers and about 50 clocks.
__device__ __forceinline__ void trace_stamp(long long* trace, int lane_id, int& n) {
#ifdef GB_FA_TRACE
  if (trace && n < kTraceSlots) trace[lane_id * kTraceSlots + n++] = clock64();
#else
  (void)trace; (void)lane_id; (void)n;
#endif
}

__device__ __forceinline__ uint32_t pack16(float a, float b, int bf) {
  return bf ? pack_bf16(a, b) : pack_f16(a, b);
}

// Stores `n` fp32 values (n multiple of 8) as 16-bit to a 16-byte aligned row.
template <int N>
__device__ __forceinline__ void store_row16(void* dst, const float* v, int bf) {
#pragma unroll
  for (int j = 0; j < N; j += 8) {
    uint4 o;
    o.x = pack16(v[j], v[j + 1], bf);
    o.y = pack16(v[j + 2], v[j + 3], bf);
    o.z = pack16(v[j + 4], v[j + 5], bf);
    o.w = pack16(v[j + 6], v[j + 7], bf);
    *reinterpret_cast<uint4*>((uint16_t*)dst + j) = o;
  }
}

// The same for a row of which only `ncols` columns (a multiple of 8, counted from this pointer)
// exist in memory: head sizes below the kernel's compile-time HD.
template <int N>
__device__ __forceinline__ void store_row16_lim(void* dst, const float* v, int bf, int ncols) {
  if (ncols >= N) {
    store_row16<N>(dst, v, bf);
    return;
  }
#pragma unroll
  for (int j = 0; j < N; j += 8) {
    if (j < ncols) {
      uint4 o;
      o.x = pack16(v[j], v[j + 1], bf);
      o.y = pack16(v[j + 2], v[j + 3], bf);
      o.z = pack16(v[j + 4], v[j + 5], bf);
      o.w = pack16(v[j + 6], v[j + 7], bf);
      *reinterpret_cast<uint4*>((uint16_t*)dst + j) = o;
    }
  }
}

// Two packed fp32 products.
__device__ __forceinline__ unsigned long long fmul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long pair(uint32_t lo, uint32_t hi) { return (unsigned long long)hi << 32 | lo; }
__device__ __forceinline__ float lo_of(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long fadd2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long pairf(float lo, float hi) { return pair(__float_as_uint(lo), __float_as_uint(hi)); }

template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t addr, uint32_t (&r)[N]) {
  if constexpr (N == 32) tmem_ld32(addr, r);
  else tmem_ld16(addr, r);
}
template <int N>
__device__ __forceinline__ void tmem_st_cols(uint32_t addr, const uint32_t (&r)[N]) {
  if constexpr (N == 16) {
    tmem_st16(addr, r);
  } else {
    static_assert(N == 8, "columns");
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
  }
}

template <bool BF>
__device__ __forceinline__ uint32_t pack16t(float a, float b) {
  return BF ? pack_bf16(a, b) : pack_f16(a, b);
}

constexpr int BKF = 64;  // key rows per forward sub-tile

// Forward tiling: 128 query rows per CTA, keys in 64-row sub-tiles.  Two score buffers of 64
// columns and the output accumulator need 128 + HD <= 256 TMEM columns, and the shared
// memory of one CTA stays under half an SM, so two CTAs share an SM: while the softmax warps
// of one are busy, the tensor core serves the other.  With one score buffer a head of 64 takes 128 columns, and four CTAs
// share the SM: four softmax warps per scheduler instead of two, each with a longer chain (the next scores follow this
// sub-tile's P V), which pays once there are CTAs enough.
template <int HD, int NBUF_>
struct FwdCfg {
  static constexpr int CH = HD / 64;                   // 64-column chunks per row
  static constexpr int Q_BYTES = CH * BQ * 128;        // the resident query tile
  static constexpr int SUB_BYTES = CH * BKF * 128;     // one K or V sub-tile
  static constexpr int NBUF = NBUF_;                   // score buffers
  static constexpr int CTAS_PER_SM = NBUF == 1 ? 4 : 2;
  static_assert(NBUF == 2 || HD == 64, "four CTAs share TMEM");
  static constexpr int STAGES = NBUF == 2 && HD == 64 ? 3 : 2;
  static constexpr int SMEM_BYTES = Q_BYTES + 2 * STAGES * SUB_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = NBUF == 1 ? 128 : 256;
  static constexpr int COL_S = 0, COL_O = NBUF * BKF;
};

template <int HD, bool BF, int NBUF>
__global__ void __launch_bounds__(kFwdThreads, FwdCfg<HD, NBUF>::CTAS_PER_SM)
fa_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const AttnArgs args) {
  using C = FwdCfg<HD, NBUF>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + C::Q_BYTES;                   // [STAGES]
  uint8_t* sV = sK + C::STAGES * C::SUB_BYTES;     // [STAGES]
  uint64_t* bars = (uint64_t*)(sV + C::STAGES * C::SUB_BYTES);
  uint64_t* q_full = bars;                    // 1
  uint64_t* k_full = bars + 1;                // STAGES
  uint64_t* k_empty = k_full + C::STAGES;     // STAGES
  uint64_t* v_full = k_empty + C::STAGES;     // STAGES
  uint64_t* v_empty = v_full + C::STAGES;     // STAGES
  uint64_t* s_full = v_empty + C::STAGES;     // 2
  uint64_t* p_full = s_full + 2;              // 2
  uint64_t* pv_done = p_full + 2;             // 2
  uint32_t* tmem_slot = (uint32_t*)(pv_done + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_q_tiles = (args.Sq + BQ - 1) / BQ;
  int rank, h, b;
  block_of(args, rank, h, b);
  const int q_tile = args.causal ? num_q_tiles - 1 - rank : rank;   // heavy (late) query tiles first when causal
  const int q0 = q_tile * BQ;
  int n_kv = (args.Sk + BKF - 1) / BKF;
  if (args.causal) n_kv = min(n_kv, (q_tile + 1) * (BQ / BKF));

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < C::STAGES; i++) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);  // one arrival per softmax warp
      mbar_init(&pv_done[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  } else if (warp == 2 && lane < 4) {
    tma_prefetch_desc(lane == 0 ? &tmK : lane == 1 ? &tmQ : lane == 2 ? &tmV : &tmO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(q_full, C::Q_BYTES);
#pragma unroll
      for (int c = 0; c < C::CH; c++) tma_load_4d(sQ + c * BQ * 128, &tmQ, q_full, c * 64, q0, h, b);
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_kv; j++) {
        if (!mbar_wait(&k_empty[st], ph ^ 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 1)) break;
        mbar_expect_tx(&k_full[st], C::SUB_BYTES);
#pragma unroll
        for (int c = 0; c < C::CH; c++)
          tma_load_4d(sK + st * C::SUB_BYTES + c * BKF * 128, &tmK, &k_full[st], c * 64, j * BKF, h, b);
        if (!mbar_wait(&v_empty[st], ph ^ 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 2)) break;
        mbar_expect_tx(&v_full[st], C::SUB_BYTES);
#pragma unroll
        for (int c = 0; c < C::CH; c++)
          tma_load_4d(sV + st * C::SUB_BYTES + c * BKF * 128, &tmV, &v_full[st], c * 64, j * BKF, h, b);
        if (++st == C::STAGES) { st = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t fmt = BF ? 1u : 0u;
      const uint32_t idesc_s = make_idesc(1u, fmt, false, false, BQ, BKF);
      const uint32_t idesc_o = make_idesc(1u, fmt, false, true, BQ, HD);
      const uint32_t qa = smem_u32(sQ);
      bool ok = mbar_wait(q_full, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 3);
      int st_s = 0;
      uint32_t ph_s = 0;
      auto issue_s = [&](int j) {
        if (!mbar_wait(&k_full[st_s], ph_s, abort_flag, args.status, ST_ATTN_TIMEOUT, 4)) return false;
        tc_fence_after();
        const uint32_t ka = smem_u32(sK + st_s * C::SUB_BYTES);
        const uint32_t d = tmem_base + C::COL_S + j % C::NBUF * BKF;
#pragma unroll
        for (int k = 0; k < HD / 16; k++)
          tc_mma_f16(d, make_smem_desc_sw128(qa + (k / 4) * (BQ * 128) + (k % 4) * 32, 16, 1024),
                     make_smem_desc_sw128(ka + (k / 4) * (BKF * 128) + (k % 4) * 32, 16, 1024), idesc_s, k != 0);
        tc_commit(&k_empty[st_s]);
        tc_commit(&s_full[j % C::NBUF]);
        if (++st_s == C::STAGES) { st_s = 0; ph_s ^= 1; }
        return true;
      };
      if (ok && n_kv > 0) ok = issue_s(0);
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_kv && ok; j++) {
        if (C::NBUF == 2 && j + 1 < n_kv) {       // two buffers: the next scores before this sub-tile's P is waited for
          ok = issue_s(j + 1);
          if (!ok) break;
        }
        const int sb = j % C::NBUF;
        ok = mbar_wait(&p_full[sb], (j / C::NBUF) & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 5);
        if (!ok) break;
        ok = mbar_wait(&v_full[st], ph, abort_flag, args.status, ST_ATTN_TIMEOUT, 6);
        if (!ok) break;
        tc_fence_after();
        const uint32_t va = smem_u32(sV + st * C::SUB_BYTES);
        const uint32_t p_tmem = tmem_base + C::COL_S + sb * BKF;
        const uint32_t d = tmem_base + C::COL_O;
#pragma unroll
        for (int k = 0; k < BKF / 16; k++) {
          // V is the MN-major B operand: 64-wide d chunks are BKF*128 B apart, 8-row groups
          // 1024 B apart, one MMA step covers 16 key rows.
          tc_mma_f16_ts(d, p_tmem + (k >> 1) * 32 + (k & 1) * 8, make_smem_desc_sw128(va + k * 16 * 128, BKF * 128, 1024), idesc_o,
                        (j | k) != 0);
        }
        tc_commit(&v_empty[st]);
        tc_commit(&pv_done[sb]);
        if (++st == C::STAGES) { st = 0; ph ^= 1; }
        if (C::NBUF == 1 && j + 1 < n_kv) ok = issue_s(j + 1);
      }
    }
    __syncwarp();
  } else {
    // ---------------- softmax warps: thread = row ----------------
    // What bounds the kernel is the chain of such a warp: the exponentials of a sub-tile, 512 clocks of its scheduler, and about
    // as much again of waits, loads and hand-overs (MUFU 65 % busy at head size 64).  So the maximum is four chains, products and
    // sums are packed, and O leaves by TMA.  (Scores of the next
    // sub-tile loaded while exponentials run, or two warps to a row: slower.)  us before -> now: (16, 12, 1024, 64) causal
    // 66.0 -> 53.9, (6, 12, 1000 x 1531, 64) 51.9 -> 49.4, (8, 16, 4096, 128) causal 535 -> 502, (4, 16, 2048, 128) 79.7 -> 74.5.
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;  // row inside the tile
    const int qrow = q0 + r;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const unsigned long long sl2 = pairf(args.scale_log2, args.scale_log2);
    float m_used = -INFINITY;  // in log2 units, already scaled
    unsigned long long l2 = 0ull;   // the row sum, as two sums
    // sub-tiles entirely to the right of this warp's 32 rows (from q0 + 32 * quarter) contribute nothing: P = 0, running max
    // and sum unchanged
    const int n_live = args.causal ? min(n_kv, (q0 + quarter * 32 + 31) / BKF + 1) : n_kv;
    uint32_t s[C::NBUF][32];
    auto wait_scores = [&](int j) {
      const bool ready = mbar_wait(&s_full[j % C::NBUF], (j / C::NBUF) & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 7);
      tc_fence_after();
      return ready;
    };
    auto scores_at = [&](int j) { return lane_addr + C::COL_S + j % C::NBUF * BKF; };
    auto give_p = [&](int j) {
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[j % C::NBUF]);
    };
    bool ok = true;
    for (int j = 0; j < n_live; j++) {
      ok = wait_scores(j);
      if (!ok) break;
      const uint32_t s_addr = scores_at(j);
      const int kv0 = j * BKF;
      const bool masked = (args.causal && kv0 + BKF - 1 > q0 + quarter * 32) || kv0 + BKF > args.Sk;
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      auto load_half = [&](int g) { tmem_ld32(s_addr + g * 32, s[C::NBUF == 2 ? g : 0]); };
      auto mask_half = [&](int g) {
        if (masked) {
#pragma unroll
          for (int c = 0; c < 32; c++)
            if (kv0 + g * 32 + c >= args.Sk || (args.causal && kv0 + g * 32 + c > qrow)) s[C::NBUF == 2 ? g : 0][c] = 0xff800000u;
        }
      };
      if (C::NBUF == 2) { load_half(0); load_half(1); }
#pragma unroll
      for (int g = 0; g < 2; g++) {
        if (C::NBUF == 1) load_half(g);
        if (C::NBUF == 1 || g == 0) tmem_ld_wait();
        mask_half(g);
#pragma unroll
        for (int c = 0; c < 32; c++) mx[c & 3] = fmaxf(mx[c & 3], __uint_as_float(s[C::NBUF == 2 ? g : 0][c]));
      }
      float m_new = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * args.scale_log2);
      if (m_new == -INFINITY) m_new = 0.f;
      // rescale O only when the running max moved by more than 8 (a factor 256)
      const bool need = (m_new - m_used) > 8.f;
      if (__any_sync(0xffffffffu, need)) {
        float alpha = 1.f;
        if (need) {
          alpha = (m_used == -INFINITY) ? 0.f : exp2f(m_used - m_new);
          m_used = m_new;
          l2 = fmul2(l2, pairf(alpha, alpha));
        }
        if (j > 0) {
          ok = mbar_wait(&pv_done[(j - 1) % C::NBUF], ((j - 1) / C::NBUF) & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 8);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < HD / 16; c++) {
            uint32_t ro[16];
            tmem_ld16(lane_addr + C::COL_O + c * 16, ro);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i++) ro[i] = __float_as_uint(__uint_as_float(ro[i]) * alpha);
            tmem_st16(lane_addr + C::COL_O + c * 16, ro);
          }
          tmem_st_wait();
        }
      }
      const unsigned long long nm2 = pairf(-m_used, -m_used);
      // the second half first: it is the one in registers where they hold one.  P goes over the columns that its scores came from.
#pragma unroll
      for (int g = 1; g >= 0; g--) {
        if (C::NBUF == 1 && g == 0) {
          load_half(0);
          tmem_ld_wait();
          mask_half(0);
        }
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const uint32_t* x2 = s[C::NBUF == 2 ? g : 0];
          const unsigned long long x = ffma2(pair(x2[2 * i], x2[2 * i + 1]), sl2, nm2);
          const float p0 = exp2f(lo_of(x)), p1 = exp2f(hi_of(x));
          l2 = fadd2(l2, pairf(p0, p1));
          pk[i] = pack16t<BF>(p0, p1);
        }
        tmem_st16(s_addr + g * 32, pk);
      }
      give_p(j);
    }
    for (int j = n_live; j < n_kv && ok; j++) {
      ok = wait_scores(j);
      if (!ok) break;
      uint32_t zero[16];
#pragma unroll
      for (int i = 0; i < 16; i++) zero[i] = 0u;
      tmem_st16(scores_at(j), zero);
      tmem_st16(scores_at(j) + 32, zero);
      give_p(j);
    }
    if (ok && n_kv > 0)
      ok = mbar_wait(&pv_done[(n_kv - 1) % C::NBUF], ((n_kv - 1) / C::NBUF) & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 9);
    if (ok) {
      tc_fence_after();
      const float l = lo_of(l2) + hi_of(l2);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // through the query tile, which every MMA has read by now, and a TMA store of this warp's rows (rows and columns behind
      // the tensor's ends are clipped)
#pragma unroll
      for (int c = 0; c < HD / 32; c++) {
        uint32_t ro[32];
        if (n_kv > 0) {
          tmem_ld32(lane_addr + C::COL_O + c * 32, ro);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; i++) ro[i] = 0;
        }
        const uint32_t row = smem_u32(sQ) + c / 2 * (BQ * 128) + (uint32_t)r * 128u;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; i++)
            w[i] = pack16t<BF>(__uint_as_float(ro[8 * q + 2 * i]) * inv, __uint_as_float(ro[8 * q + 2 * i + 1]) * inv);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + (((uint32_t)(c % 2 * 4 + q) ^ ((uint32_t)r & 7u)) << 4)),
                       "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && q0 + quarter * 32 < args.Sq) {
#pragma unroll
        for (int c = 0; c < C::CH; c++)
          if (c * 64 < args.D) tma_store_4d(&tmO, sQ + c * BQ * 128 + quarter * 32 * 128, c * 64, q0 + quarter * 32, h, b);
        tma_store_commit();
      }
      if (qrow < args.Sq && args.LSE) {
        // natural-log LSE of the scaled scores
        args.LSE[((long long)b * args.H + h) * args.Sq + qrow] =
            l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
      if (lane == 0) tma_store_wait_read<0>();   // shared memory must outlive the stores that read from it
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// Delta[b,h,q] = sum_d dO[b,q,h,d] * O[b,q,h,d]  (fp32), one warp per row
template <typename T>
__global__ void fa_delta_kernel(const T* __restrict__ O, const T* __restrict__ dO,
                                float* __restrict__ delta, int B, int H, int S, int D,
                                long long o_sb, long long o_ss, long long o_sh, long long g_sb,
                                long long g_ss, long long g_sh) {
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long total = (long long)B * H * S;
  for (long long i = (long long)blockIdx.x * warps + warp; i < total; i += (long long)gridDim.x * warps) {
    const int q = (int)(i % S);
    const int h = (int)((i / S) % H);
    const int b = (int)(i / ((long long)S * H));
    const T* o = O + b * o_sb + q * o_ss + h * o_sh;
    const T* g = dO + b * g_sb + q * g_ss + h * g_sh;
    float s = 0.f;
    for (int d = lane; d < D; d += 32) s += (float)o[d] * (float)g[d];
    s = warp_sum(s);
    if (lane == 0) delta[i] = s;
  }
}


// The same for 16-byte aligned rows of D = 8 * TPR elements: TPR threads per row, one 16-byte load of O and of dO each for four rows
// at a time.  Rows are visited in (b, s, h) order so that neighbouring threads read neighbouring memory; I: the type that rows
// are counted in (the 64-bit divisions of one row at a time kept the loads waiting: (8, 16, 4096, 128) 72 -> 56 us, (16, 12, 1024,
// 64) 15.2 -> 10.2).
template <typename T, int TPR, typename I>
__global__ void __launch_bounds__(256)
fa_delta_vec_kernel(const T* __restrict__ O, const T* __restrict__ dO, float* __restrict__ delta, int B,
                    int H, int S, long long o_sb, long long o_ss, long long o_sh, long long g_sb,
                    long long g_ss, long long g_sh) {
  constexpr int R = 4;
  const I total = (I)B * (I)H * (I)S;
  const int sub = threadIdx.x % TPR;
  constexpr int RPB = 256 / TPR;  // rows per CTA and load; every thread of the CTA runs the same trip count
  for (I base = (I)blockIdx.x * (RPB * R); base < total; base += (I)gridDim.x * (RPB * R)) {
    uint4 uo[R], ug[R];
    I at[R];
#pragma unroll
    for (int k = 0; k < R; k++) {
      const I i = base + (I)(k * RPB + threadIdx.x / TPR);
      const I ii = i < total ? i : 0;
      const I bs = ii / (I)H, h = ii - bs * (I)H, b = bs / (I)S, q = bs - b * (I)S;
      at[k] = i < total ? (b * (I)H + h) * (I)S + q : total;
      uo[k] = *reinterpret_cast<const uint4*>(O + (long long)b * o_sb + (long long)q * o_ss + (long long)h * o_sh + sub * 8);
      ug[k] = *reinterpret_cast<const uint4*>(dO + (long long)b * g_sb + (long long)q * g_ss + (long long)h * g_sh + sub * 8);
    }
#pragma unroll
    for (int k = 0; k < R; k++) {
      const T* eo = reinterpret_cast<const T*>(&uo[k]);
      const T* eg = reinterpret_cast<const T*>(&ug[k]);
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 8; j++) s += (float)eo[j] * (float)eg[j];
#pragma unroll
      for (int o = TPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (at[k] < total && sub == 0) delta[at[k]] = s;
    }
  }
}

// ---------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------
constexpr int BSUB = 64;                  // rows of one streamed sub-tile

// Tiling of the dQ kernel that computes the scores itself.  The resident operand pair is a 128-row tile; the streamed pair comes in
// 64-row sub-tiles through a ring of NS stages.  Scores and dP of a sub-tile are 128 x 64
// fp32 blocks in TMEM, double buffered, so the tensor core computes sub-tile i+1 (and the
// accumulations of sub-tile i-1) while the elementwise warps work on sub-tile i.  The
// elementwise warps form two groups of eight; group g owns TMEM buffer g and every second
// sub-tile, so the TMEM round trips of one group hide behind the arithmetic of the other.
template <int HD>
struct BwdCfg {
  static constexpr int CH = HD / 64;
  static constexpr int TILE_BYTES = CH * 128 * 128;
  static constexpr int SUB_BYTES = CH * BSUB * 128;
  static constexpr int NS = 4;
  static constexpr int SMEM_BYTES = 2 * TILE_BYTES + NS * 2 * SUB_BYTES + 1024 + 256;      // of the dQ kernel
  // head_dim 64: one S/dP buffer, eight elementwise warps, 256 TMEM columns and < 113 KB of
  // shared memory, so TWO CTAs share an SM and hide each other's serial chain (S/dP MMAs ->
  // elementwise -> accumulation MMAs) as well as each other's start-up and epilogue.
  // head_dim 128: the accumulators alone need 256 columns, so one CTA per SM with two S/dP
  // buffers and two groups of eight elementwise warps that own alternate sub-tiles.
  static constexpr bool DUAL = HD == 64;             // two CTAs per SM
  static constexpr int NBUF = DUAL ? 1 : 2;
  static constexpr int EW = 8 * NBUF;
  static constexpr int THREADS = 64 + EW * 32;
  static constexpr int CTAS_PER_SM = DUAL ? 2 : 1;
  static constexpr int TMEM_COLS = DUAL ? 256 : 512;
  // buffer b: scores at b*128, dP at b*128 + 64; accumulators behind them
  static constexpr int COL_ACC0 = 128 * NBUF, COL_ACC1 = COL_ACC0 + HD;
  // resident A operands kept in TMEM where the columns allow it
  static constexpr bool Q_IN_TMEM = !DUAL;
  static constexpr int COL_QT = COL_ACC0 + HD, COL_GT = COL_QT + HD / 2;
};

// K-major operand descriptor for step k (16 columns) of a [128 x HD] tile
__device__ __forceinline__ uint64_t kdesc(uint32_t base, int k) {
  return make_smem_desc_sw128(base + (k / 4) * (128 * 128) + (k % 4) * 32, 16, 1024);
}
// the same for a [64 x HD] sub-tile (64-column chunks are 64 rows apart)
__device__ __forceinline__ uint64_t kdesc_sub(uint32_t base, int k) {
  return make_smem_desc_sw128(base + (k / 4) * (BSUB * 128) + (k % 4) * 32, 16, 1024);
}
// MN-major operand descriptor for step k (16 rows) of a [64 rows x HD] sub-tile
__device__ __forceinline__ uint64_t mndesc_sub(uint32_t base, int k) {
  return make_smem_desc_sw128(base + k * 16 * 128, BSUB * 128, 1024);
}

// Copies this thread's row of a resident [128 x HD] 16-bit tile (128-byte swizzled rows in
// 64-column chunks of 128 rows) into TMEM columns [col, col + HD / 2): the layout of an A
// operand read from tensor memory, so the MMAs that use the tile stop re-reading it from
// shared memory on every step.
template <int HD>
__device__ __forceinline__ void tile_row_to_tmem(const uint8_t* tile, int r, uint32_t lane_addr, uint32_t col) {
#pragma unroll
  for (int c = 0; c < HD / 64; c++) {
    uint32_t w[32];
    const uint32_t row = smem_u32(tile + c * 128 * 128 + r * 128);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint4 u;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                   : "r"(row + (((uint32_t)j ^ ((uint32_t)r & 7u)) << 4)));
      w[4 * j] = u.x; w[4 * j + 1] = u.y; w[4 * j + 2] = u.z; w[4 * j + 3] = u.w;
    }
    tmem_st32(lane_addr + col + c * 32, w);
  }
  tmem_st_wait();
}

// The row statistics of the dK / dV kernel are added by the tensor core.  They belong to the columns of S^T and dP^T, so that
// every thread would need all of them: 64 values per sub-tile and warp, and shared memory delivers one register per thread and
// clock however they are loaded (560 of 2 360 clocks per 128 x 64 block).  Instead row q of a B operand of 16 k's holds -LSE / scale
// or -Delta as three bf16 parts, 24 bits, and one MMA step with an A operand of ones at their places adds it to every row of S^T or
// dP^T.  LSE and Delta have an operand each: what is infinite in one would be NaN in the other's product with the zeros at its
// places.  This is the row's first eight k's (the others are zero).  A value that is not finite has one part; a finite one that
// would round to infinity in bf16 is cut and keeps the rest in the other parts.
__device__ __forceinline__ uint4 three_parts(float x) {
  const bool fin = (__float_as_uint(x) & 0x7fffffffu) < 0x7f800000u;
  const float top = __uint_as_float(0x7f7f0000u);                 // bf16's largest value
  const __nv_bfloat16 h = __float2bfloat16_rn(fin ? fminf(fmaxf(x, -top), top) : x);
  const float r = fin ? x - __bfloat162float(h) : 0.f;
  const __nv_bfloat16 m = __float2bfloat16_rn(r);
  const __nv_bfloat16 l = __float2bfloat16_rn(r - __bfloat162float(m));
  return make_uint4(__bfloat16_as_ushort(h) | (uint32_t)__bfloat16_as_ushort(m) << 16, __bfloat16_as_ushort(l), 0u, 0u);
}
// Rows past the end and rows without any key (LSE = -inf) get a statistic that makes their probabilities 0.
__device__ __forceinline__ uint4 lse_parts(float lse, float inv_scale) {
  float x = -(lse == -INFINITY ? 1e30f : lse) * inv_scale;
  if (fabsf(x) > 1e37f) x = copysignf(1e37f, x);     // (a NaN stays one)
  return three_parts(x);
}

// dK / dV: one CTA per 128-key tile; streams 64-row query sub-tiles.  Works in the
// transposed domain (rows = keys) so that P^T is an A operand in TMEM, and dS^T one in shared memory, from where a TMA store also
// takes it to the dQ kernel (64-byte row stores by the threads took 55 clocks of the memory pipe per instruction, 890 of
// 2 360 per block).
//
// One S^T and one dP^T block of 128 x 64 in TMEM, handed to and fro in two half steps, so that the tensor core and the elementwise
// warps work at the same time on one sub-tile and the next:
//     tensor core   dV += P^T(i) dO(i), S^T(i + 1)  |  dK += dS^T(i) Q(i), dP^T(i + 1)
//     elementwise   dS^T(i) from P and dP^T(i)      |  P^T(i + 1) from S^T(i + 1)
// What bounds it at head size 128 is the shared memory that feeds the tensor core (128 bytes a clock): with K and V as A operands
// there a block moved 204 KB of it, 1 630 clocks for 1 090 of multiply-adds.  K and V therefore live in TMEM, which the single
// S^T / dP^T pair leaves room for: 140 KB.  At head size 64 two CTAs share an SM (and hide each other's start and end), each
// with half of TMEM, and K and V stay in shared memory.
// What is left is the chain of an elementwise warp: per 128 x 64 block 1.01 us at 128 (1.37 with both gathered and stored by
// the threads and two S^T / dP^T buffers), 0.67 us at 64 (1.00), where 0.57 and 0.31 are multiply-adds and 0.27 exponentials.
// us: (8, 16, 4096, 128) causal 1 343 -> 1 100; (16, 12, 1024, 64) causal 147 -> 90; (6, 12, 1000 x 1531, 64) fp16 150 -> 84.
template <int HD>
struct KvCfg {
  static constexpr bool DUAL = HD == 64;             // two CTAs per SM
  static constexpr int CH = HD / 64;
  static constexpr int TILE_BYTES = CH * 128 * 128;
  static constexpr int SUB_BYTES = CH * BSUB * 128;
  static constexpr int NS = 3;
  static constexpr int EW = DUAL ? 8 : 16;           // elementwise warps
  static constexpr int CW = 4 * BSUB / EW;           // query columns of one of them: a quarter of the key rows, all EW / 4 groups
  static constexpr int THREADS = 96 + EW * 32;       // TMA, MMA and store warps
  static constexpr int CTAS_PER_SM = DUAL ? 2 : 1;
  // row statistics (64 rows of 16 bytes for LSE and for Delta of each stage, and once the zeros behind them), the A operand that adds
  // them, the tile through which dS^T leaves
  static constexpr int STAT_ROWS = BSUB * 16, STAT_BYTES = (2 * NS + 1) * STAT_ROWS, ONES_BYTES = 1024, OUT_BYTES = 128 * 128;
  static constexpr int SMEM_BYTES = 2 * TILE_BYTES + NS * 2 * SUB_BYTES + STAT_BYTES + ONES_BYTES + OUT_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = DUAL ? 256 : 512;
  static constexpr int COL_S = 0, COL_DP = BSUB, COL_ACC0 = 2 * BSUB, COL_ACC1 = COL_ACC0 + HD;
  static constexpr bool KV_IN_TMEM = !DUAL;
  static constexpr int COL_K = COL_ACC1 + HD, COL_V = COL_K + HD / 2;
  static_assert((KV_IN_TMEM ? COL_V + HD / 2 : COL_K) <= TMEM_COLS, "TMEM");
};

template <int HD, bool BF>
__global__ void __launch_bounds__(KvCfg<HD>::THREADS, KvCfg<HD>::CTAS_PER_SM)
fa_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                  const __grid_constant__ CUtensorMap tmDS, const __grid_constant__ CUtensorMap tmdK,
                  const __grid_constant__ CUtensorMap tmdV, const AttnArgs args) {
  using C = KvCfg<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::TILE_BYTES;
  uint8_t* ring = sV + C::TILE_BYTES;                 // [NS] x {Q sub-tile, dO sub-tile}
  uint8_t* sStat = ring + C::NS * 2 * C::SUB_BYTES;   // [NS][LSE, Delta] rows, then rows of zeros
  uint8_t* sOnes = sStat + C::STAT_BYTES;             // eight rows: ones for the three parts
  uint8_t* sOut = sOnes + C::ONES_BYTES;              // 128 key rows x 64 queries of dS^T
  uint64_t* bars = (uint64_t*)(sOut + C::OUT_BYTES);
  uint64_t* kv_full = bars;                 // 1
  uint64_t* q_full = bars + 1;              // NS
  uint64_t* q_empty = q_full + C::NS;       // NS
  uint64_t* s_full = q_empty + C::NS;       // the rest: 1 each, completed once per sub-tile
  uint64_t* dp_full = s_full + 1;
  uint64_t* p_full = s_full + 2;
  uint64_t* ds_full = s_full + 3;
  uint64_t* out_empty = s_full + 4;
  uint64_t* acc_done = s_full + 5;          // once
  uint64_t* a_ready = s_full + 6;           // once: K and V copied into TMEM
  uint32_t* tmem_slot = (uint32_t*)(a_ready + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int kv_tile, h, b;                        // early key tiles are the longest when causal
  block_of(args, kv_tile, h, b);
  const int kv0 = kv_tile * BKV;
  const int num_sub = (args.Sq + BSUB - 1) / BSUB;
  const int i_begin = args.causal ? kv_tile * (BKV / BSUB) : 0;
  const int n_it = max(num_sub - i_begin, 0);

  const float* lse = args.LSE + ((long long)b * args.H + h) * args.Sq;
  const float* delta = args.Delta + ((long long)b * args.H + h) * args.Sq;
  float nl[2], nd[2];
  auto read_stats = [&](int it) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int q = (i_begin + it) * BSUB + lane + 32 * i;
      nl[i] = q < args.Sq ? __ldg(lse + q) : -INFINITY;
      nd[i] = q < args.Sq ? __ldg(delta + q) : 0.f;
    }
  };
  if (warp == 0) read_stats(0);                // (used by the producer warp only)
  auto load_stage = [&](int it, int st) {      // Q and dO of a sub-tile, by one thread
    const int q0 = (i_begin + it) * BSUB;
    mbar_expect_tx(&q_full[st], 2 * C::SUB_BYTES);
    uint8_t* sQ = ring + st * 2 * C::SUB_BYTES;
    uint8_t* sdO = sQ + C::SUB_BYTES;
#pragma unroll
    for (int c = 0; c < C::CH; c++) {
      tma_load_4d(sQ + c * BSUB * 128, &tmQ, &q_full[st], c * 64, q0, h, b);
      tma_load_4d(sdO + c * BSUB * 128, &tmdO, &q_full[st], c * 64, q0, h, b);
    }
  };
  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < C::NS; i++) {
      mbar_init(&q_full[i], 1 + 32);  // the TMA transaction + the 32 lanes that stage the row statistics
      mbar_init(&q_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, C::EW);
    mbar_init(ds_full, C::EW);
    mbar_init(out_empty, args.dS ? 2 : 1);   // the MMAs that read the tile and its TMA store
    mbar_init(acc_done, 1);
    mbar_init(a_ready, 8);
    *abort_flag = 0;
    mbar_fence_init();
    // the loads of the tile and of the first stages start before anything else is ready
    fence_proxy_async_smem();
    mbar_expect_tx(kv_full, 2 * C::TILE_BYTES);
#pragma unroll
    for (int c = 0; c < C::CH; c++) {
      tma_load_4d(sK + c * 128 * 128, &tmK, kv_full, c * 64, kv0, h, b);
      tma_load_4d(sV + c * 128 * 128, &tmV, kv_full, c * 64, kv0, h, b);
    }
    if (n_it > 0) load_stage(0, 0);
  } else if (warp == 2) {
    if (lane < 4) tma_prefetch_desc(lane == 0 ? &tmK : lane == 1 ? &tmV : lane == 2 ? &tmQ : &tmdO);
    else if (lane < 7) tma_prefetch_desc(lane == 4 ? &tmdK : lane == 5 ? &tmdV : &tmDS);
  }
  if (threadIdx.x < 64) {
    const uint32_t row = threadIdx.x >> 3, chunk = (threadIdx.x & 7u) ^ row;      // 16-byte chunk before the swizzle
    constexpr uint32_t one = 0x3f80u;
    reinterpret_cast<uint4*>(sOnes)[threadIdx.x] = chunk == 0u ? make_uint4(one | one << 16, one, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4*>(sStat + 2 * C::NS * C::STAT_ROWS)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
  }
  fence_proxy_async_smem();
  if (warp == 1) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---- producer: TMA for the sub-tiles (lane 0), row statistics by all lanes, read one sub-tile ahead ----
    if (lane == 0)
      for (int it = 1; it < min(n_it, C::NS); it++) load_stage(it, it);
    int st = 0;
    uint32_t ph = 0;
    for (int it = 0; it < n_it; it++) {
      const float l[2] = {nl[0], nl[1]}, d[2] = {nd[0], nd[1]};
      read_stats(it + 1);
      if (it >= C::NS) {
        int ok = 1;
        if (lane == 0) ok = mbar_wait(&q_empty[st], ph ^ 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 11);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        if (lane == 0) load_stage(it, st);
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        uint4* row = reinterpret_cast<uint4*>(sStat + 2 * st * C::STAT_ROWS) + lane + 32 * i;
        row[0] = lse_parts(l[i], args.inv_scale);
        row[C::STAT_ROWS / 16] = three_parts(-d[i]);
      }
      fence_proxy_async_smem();
      mbar_arrive(&q_full[st]);
      if (++st == C::NS) { st = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t fmt = BF ? 1u : 0u;
      const uint32_t idesc_s = make_idesc(1u, fmt, false, false, 128, BSUB);
      const uint32_t idesc_acc = make_idesc(1u, fmt, false, true, 128, HD);
      const uint32_t idesc_stat = make_idesc(1u, 1u, false, false, 128, BSUB);
      const uint32_t ones = smem_u32(sOnes), stat = smem_u32(sStat);
      bool ok = mbar_wait(kv_full, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 12);
      if (ok && C::KV_IN_TMEM) {
        ok = mbar_wait(a_ready, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 18);
        tc_fence_after();
      }
      // S^T = K Q^T - LSE / scale (tile sK, sub-tile at 0) or dP^T = V dO^T - Delta (sV, second sub-tile) of the sub-tile in a stage
      auto issue = [&](int st, int which) {
        const uint32_t sub = smem_u32(ring + st * 2 * C::SUB_BYTES) + which * C::SUB_BYTES;
        const uint32_t tile = smem_u32(sK) + which * C::TILE_BYTES;
        const uint32_t d = tmem_base + (which ? C::COL_DP : C::COL_S);
#pragma unroll
        for (int k = 0; k < HD / 16; k++) {
          if (C::KV_IN_TMEM) tc_mma_f16_ts(d, tmem_base + (which ? C::COL_V : C::COL_K) + k * 8, kdesc_sub(sub, k), idesc_s, k != 0);
          else tc_mma_f16(d, kdesc(tile, k), kdesc_sub(sub, k), idesc_s, k != 0);
        }
        const int at = (2 * st + which) * C::STAT_ROWS;
        tc_mma_f16(d, make_smem_desc_sw128(ones, 16, 0), make_smem_desc_plain(stat + at, 2 * C::NS * C::STAT_ROWS - at, 128), idesc_stat, 1u);
        tc_commit(which ? dp_full : s_full);
      };
      // dV += P^T dO (which = 0) or dK += dS^T Q (1).  P^T: each elementwise warp left CW / 2 packed columns at the start of its
      // own CW, so a step of 16 queries reads from there; dS^T: from the tile in shared memory
      auto accumulate = [&](int st, int which, bool first) {
        const uint32_t sub = smem_u32(ring + st * 2 * C::SUB_BYTES) + (which ? 0 : C::SUB_BYTES);
        const uint32_t d = tmem_base + (which ? C::COL_ACC1 : C::COL_ACC0);
#pragma unroll
        for (int k = 0; k < BSUB / 16; k++) {
          if (which) tc_mma_f16(d, kdesc(smem_u32(sOut), k), mndesc_sub(sub, k), idesc_acc, !first || k != 0);
          else tc_mma_f16_ts(d, tmem_base + C::COL_S + k * 16 / C::CW * C::CW + k * 16 % C::CW / 2, mndesc_sub(sub, k), idesc_acc, !first || k != 0);
        }
      };
      long long* tr = (blockIdx.x | blockIdx.y | blockIdx.z) == 0 ? args.trace : nullptr;
      int ntr = 0;
      trace_stamp(tr, 0, ntr);
      if (ok && n_it > 0) {
        ok = mbar_wait(&q_full[0], 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 13);
        if (ok) {
          tc_fence_after();
          issue(0, 0);
          issue(0, 1);
        }
      }
      int st = 0, nst = 1;
      uint32_t nph = 0;        // of the next sub-tile's stage
      for (int it = 0; it < n_it && ok; it++) {
        const uint32_t ph = it & 1;
        const bool more = it + 1 < n_it;
        ok = mbar_wait(p_full, ph, abort_flag, args.status, ST_ATTN_TIMEOUT, 14);
        if (!ok) break;
        trace_stamp(tr, 0, ntr);  // P ready
        tc_fence_after();
        accumulate(st, 0, it == 0);
        if (more) {
          ok = mbar_wait(&q_full[nst], nph, abort_flag, args.status, ST_ATTN_TIMEOUT, 13);
          if (!ok) break;
          tc_fence_after();
          issue(nst, 0);
        }
        ok = mbar_wait(ds_full, ph, abort_flag, args.status, ST_ATTN_TIMEOUT, 20);
        if (!ok) break;
        trace_stamp(tr, 0, ntr);  // dS ready
        tc_fence_after();
        accumulate(st, 1, it == 0);
        tc_commit(&q_empty[st]);
        tc_commit(out_empty);
        if (more) issue(nst, 1);
        else tc_commit(acc_done);
        st = nst;
        if (++nst == C::NS) { nst = 0; nph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 2 + C::EW) {
    // ---- dS^T out: one TMA store of 128 rows x 128 bytes per sub-tile ----
    if (args.dS && elect_one()) {
      for (int it = 0; it < n_it; it++) {
        if (!mbar_wait(ds_full, it & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 27)) break;
        tma_store_3d(&tmDS, sOut, (i_begin + it) * BSUB, kv0, b * args.H + h);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(out_empty);
      }
      tma_store_wait_read<0>();   // shared memory must outlive the stores that read from it (they complete behind the CTA)
    }
    __syncwarp();
  } else {
    constexpr int CW = C::CW;
    const int e = warp - 2;
    const int cg = e >> 2;                   // which CW of the sub-tile's 64 query columns
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;       // key row inside the tile
    const int kvrow = kv0 + r;
    const bool row_dead = kvrow >= args.Sk;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + C::COL_S + cg * CW, dp_addr = lane_addr + C::COL_DP + cg * CW;
    bool ok = true;
    if (C::KV_IN_TMEM && cg < 2) {
      ok = mbar_wait(kv_full, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 19);
      if (ok) {
        tile_row_to_tmem<HD>(cg == 0 ? sK : sV, r, lane_addr, cg == 0 ? C::COL_K : C::COL_V);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_ready);
      }
    }
    long long* tr = ((blockIdx.x | blockIdx.y | blockIdx.z) == 0 && (e & 7) == 0 && lane == 0) ? args.trace : nullptr;
    const int tl = 1 + (e >> 3);
    int ntr = 0;
    const unsigned long long sl2 = pairf(args.scale_log2, args.scale_log2);
    const unsigned long long sc2 = pairf(args.scale, args.scale);
    const uint32_t out_row = smem_u32(sOut) + (uint32_t)r * 128u;
    for (int it = 0; it < n_it; it++) {
      const uint32_t ph = it & 1;
      const int q0 = (i_begin + it) * BSUB + cg * CW;  // first query column of this thread
      // The warp's 32 key rows against its CW query columns: entirely above the diagonal (everything masked: zeros, no
      // arithmetic), entirely on or below it (no masking), or a block that the diagonal crosses (per-element test).
      const int rel = kv0 + quarter * 32 - q0;  // first key row minus first query column
      const bool all_masked = args.causal && rel > CW - 1;
      const bool masked = __any_sync(0xffffffffu, row_dead) || (args.causal && rel + 31 > 0);
      uint32_t in[CW], pk[CW / 2];
      float pr[CW];
      trace_stamp(tr, tl, ntr);
      ok = mbar_wait(s_full, ph, abort_flag, args.status, ST_ATTN_TIMEOUT, 15);
      if (!ok) break;
      trace_stamp(tr, tl, ntr);  // scores ready
      tc_fence_after();
      if (!all_masked) {
        tmem_ld_cols<CW>(s_addr, in);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < CW / 2; g++) {
          const unsigned long long x = fmul2(pair(in[2 * g], in[2 * g + 1]), sl2);
          pr[2 * g] = exp2f(lo_of(x));
          pr[2 * g + 1] = exp2f(hi_of(x));
        }
        if (masked) {
#pragma unroll
          for (int g = 0; g < CW; g++)
            if (row_dead || (args.causal && kvrow > q0 + g)) pr[g] = 0.f;
        }
      } else {
#pragma unroll
        for (int g = 0; g < CW; g++) pr[g] = 0.f;
      }
#pragma unroll
      for (int g = 0; g < CW / 2; g++) pk[g] = pack16t<BF>(pr[2 * g], pr[2 * g + 1]);
      // each warp overwrites only columns it has read itself
      tmem_st_cols<CW / 2>(s_addr, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      trace_stamp(tr, tl, ntr);  // P stored
      ok = mbar_wait(dp_full, ph, abort_flag, args.status, ST_ATTN_TIMEOUT, 17);
      if (!ok) break;
      trace_stamp(tr, tl, ntr);  // dP ready
      tc_fence_after();
      if (!all_masked) {
        tmem_ld_cols<CW>(dp_addr, in);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < CW / 2; g++) {
          const unsigned long long q = fmul2(pairf(pr[2 * g], pr[2 * g + 1]), fmul2(pair(in[2 * g], in[2 * g + 1]), sc2));
          pk[g] = pack16t<BF>(lo_of(q), hi_of(q));
        }
      }
      ok = mbar_wait(out_empty, ph ^ 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 30);
      if (!ok) break;
#pragma unroll
      for (int j = 0; j < CW / 8; j++)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(out_row + (((uint32_t)(cg * (CW / 8) + j) ^ ((uint32_t)r & 7u)) << 4)),
                     "r"(pk[4 * j]), "r"(pk[4 * j + 1]), "r"(pk[4 * j + 2]), "r"(pk[4 * j + 3])
                     : "memory");
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      trace_stamp(tr, tl, ntr);  // dS stored
    }
    if (ok && n_it > 0) ok = mbar_wait(acc_done, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 16);
    if (ok) {
      tc_fence_after();
      constexpr int W = HD * 4 / C::EW;  // columns of dV / dK per warp
      const int cw = cg * W;
      // through the ring, whose loads have all been consumed, and TMA stores of whole rows (rows and columns behind the tensors' ends
      // are clipped; 16-byte stores of 32 rows at a time took 3 000 clocks)
      static_assert(2 * C::TILE_BYTES <= C::NS * 2 * C::SUB_BYTES, "the gradient tiles reuse the ring");
#pragma unroll
      for (int o = 0; o < 2; o++) {
        uint32_t in[W];
        if (n_it > 0) {
          tmem_ld_cols<W>(lane_addr + (o ? C::COL_ACC1 : C::COL_ACC0) + cw, in);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < W; i++) in[i] = 0u;
        }
        const uint32_t row = smem_u32(ring) + o * C::TILE_BYTES + cw / 64 * (128 * 128) + (uint32_t)r * 128u;
#pragma unroll
        for (int j = 0; j < W / 8; j++) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; i++) w[i] = pack16t<BF>(__uint_as_float(in[8 * j + 2 * i]), __uint_as_float(in[8 * j + 2 * i + 1]));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + (((uint32_t)(cw % 64 / 8 + j) ^ ((uint32_t)r & 7u)) << 4)),
                       "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync 1, %0;" ::"n"(C::EW * 32) : "memory");
      if (threadIdx.x == 64) {
#pragma unroll
        for (int c = 0; c < C::CH; c++)
          if (c * 64 < args.D) {
            tma_store_4d(&tmdV, ring + c * 128 * 128, c * 64, kv0, h, b);
            tma_store_4d(&tmdK, ring + C::TILE_BYTES + c * 128 * 128, c * 64, kv0, h, b);
          }
        tma_store_commit();
        tma_store_wait_read<0>();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, C::TMEM_COLS); }
}

// dQ: one CTA per 128-row query tile; streams 64-row key sub-tiles.
template <int HD, bool BF>
__global__ void __launch_bounds__(BwdCfg<HD>::THREADS, BwdCfg<HD>::CTAS_PER_SM)
fa_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                 const AttnArgs args) {
  using C = BwdCfg<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + C::TILE_BYTES;
  uint8_t* ring = sdO + C::TILE_BYTES;  // [NS] x {K sub-tile, V sub-tile}
  uint64_t* bars = (uint64_t*)(ring + C::NS * 2 * C::SUB_BYTES);
  uint64_t* q_full = bars;                  // 1
  uint64_t* kv_full = bars + 1;             // NS
  uint64_t* kv_empty = kv_full + C::NS;     // NS
  uint64_t* sdp_full = kv_empty + C::NS;    // 2
  uint64_t* p_full = sdp_full + 2;          // 2
  uint64_t* acc_done = p_full + 2;          // 1
  uint64_t* a_ready = acc_done + 1;         // 1: Q and dO copied into TMEM
  uint32_t* tmem_slot = (uint32_t*)(a_ready + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_q_tiles = (args.Sq + BQ - 1) / BQ;
  int rank, h, b;
  block_of(args, rank, h, b);
  const int q_tile = args.causal ? num_q_tiles - 1 - rank : rank;
  const int q0 = q_tile * BQ;
  int n_sub = (args.Sk + BSUB - 1) / BSUB;
  if (args.causal) n_sub = min(n_sub, (q_tile + 1) * (BQ / BSUB));

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < C::NS; i++) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < 2; i++) { mbar_init(&sdp_full[i], 1); mbar_init(&p_full[i], 8); }
    mbar_init(acc_done, 1);
    mbar_init(a_ready, 8);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, 2 * C::TILE_BYTES);
#pragma unroll
      for (int c = 0; c < C::CH; c++) {
        tma_load_4d(sQ + c * 128 * 128, &tmQ, q_full, c * 64, q0, h, b);
        tma_load_4d(sdO + c * 128 * 128, &tmdO, q_full, c * 64, q0, h, b);
      }
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_sub; j++) {
        if (!mbar_wait(&kv_empty[st], ph ^ 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 21)) break;
        mbar_expect_tx(&kv_full[st], 2 * C::SUB_BYTES);
        uint8_t* sK = ring + st * 2 * C::SUB_BYTES;
        uint8_t* sV = sK + C::SUB_BYTES;
#pragma unroll
        for (int c = 0; c < C::CH; c++) {
          tma_load_4d(sK + c * BSUB * 128, &tmK, &kv_full[st], c * 64, j * BSUB, h, b);
          tma_load_4d(sV + c * BSUB * 128, &tmV, &kv_full[st], c * 64, j * BSUB, h, b);
        }
        if (++st == C::NS) { st = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t fmt = BF ? 1u : 0u;
      const uint32_t idesc_s = make_idesc(1u, fmt, false, false, 128, BSUB);
      const uint32_t idesc_acc = make_idesc(1u, fmt, false, true, 128, HD);
      const uint32_t qa = smem_u32(sQ), ga = smem_u32(sdO);
      bool ok = mbar_wait(q_full, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 22);
      if (ok && C::Q_IN_TMEM) {
        ok = mbar_wait(a_ready, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 28);
        tc_fence_after();
      }
      int st_s = 0;
      uint32_t ph_s = 0;
      auto issue_sdp = [&](int j) {
        if (!mbar_wait(&kv_full[st_s], ph_s, abort_flag, args.status, ST_ATTN_TIMEOUT, 23)) return false;
        tc_fence_after();
        const uint32_t ka = smem_u32(ring + st_s * 2 * C::SUB_BYTES), va = ka + C::SUB_BYTES;
        const uint32_t d = tmem_base + (j % C::NBUF) * 128;
#pragma unroll
        for (int k = 0; k < HD / 16; k++) {
          if (C::Q_IN_TMEM) {
            tc_mma_f16_ts(d, tmem_base + C::COL_QT + k * 8, kdesc_sub(ka, k), idesc_s, k != 0);       // S = Q K^T
            tc_mma_f16_ts(d + 64, tmem_base + C::COL_GT + k * 8, kdesc_sub(va, k), idesc_s, k != 0);  // dP = dO V^T
          } else {
            tc_mma_f16(d, kdesc(qa, k), kdesc_sub(ka, k), idesc_s, k != 0);
            tc_mma_f16(d + 64, kdesc(ga, k), kdesc_sub(va, k), idesc_s, k != 0);
          }
        }
        tc_commit(&sdp_full[j % C::NBUF]);
        if (++st_s == C::NS) { st_s = 0; ph_s ^= 1; }
        return true;
      };
      if (ok && n_sub > 0) ok = issue_sdp(0);
      int st = 0;
      for (int j = 0; j < n_sub && ok; j++) {
        if (C::NBUF == 2 && j + 1 < n_sub) {
          ok = issue_sdp(j + 1);
          if (!ok) break;
        }
        const int bb = j % C::NBUF;
        ok = mbar_wait(&p_full[bb], (j / C::NBUF) & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 24);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ka = smem_u32(ring + st * 2 * C::SUB_BYTES);
        const uint32_t pt = tmem_base + bb * 128 + 64;
#pragma unroll
        for (int k = 0; k < BSUB / 16; k++)  // dQ += dS K
          tc_mma_f16_ts(tmem_base + C::COL_ACC0, pt + (k >> 1) * 32 + (k & 1) * 8, mndesc_sub(ka, k), idesc_acc,
                        (j | k) != 0);
        tc_commit(&kv_empty[st]);
        if (j == n_sub - 1) tc_commit(acc_done);
        if (++st == C::NS) st = 0;
        if (C::NBUF == 1 && j + 1 < n_sub) ok = issue_sdp(j + 1);
      }
    }
    __syncwarp();
  } else {
    const int e = warp - 2;
    const int group = e >> 3;
    const int half = (e >> 2) & 1;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int qrow = q0 + r;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t my = lane_addr + group * 128 + half * 32;
    float lse2 = INFINITY, dls = 0.f;
    if (qrow < args.Sq) {
      lse2 = args.LSE[((long long)b * args.H + h) * args.Sq + qrow] * 1.4426950408889634f;
      dls = args.Delta[((long long)b * args.H + h) * args.Sq + qrow] * args.scale;
      if (lse2 == -INFINITY) lse2 = INFINITY;
    }
    bool ok = true;
    if (C::Q_IN_TMEM && group == 0) {
      // the eight warps of group 0 copy Q (half 0) and dO (half 1) into TMEM once
      ok = mbar_wait(q_full, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 29);
      if (ok) {
        tile_row_to_tmem<HD>(half == 0 ? sQ : sdO, r, lane_addr, half == 0 ? C::COL_QT : C::COL_GT);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_ready);
      }
    }
    for (int j = group; j < n_sub; j += C::NBUF) {
      ok = mbar_wait(&sdp_full[group], (j / C::NBUF) & 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 25);
      if (!ok) break;
      tc_fence_after();
      const int kv0 = j * BSUB + half * 32;  // first key column of this thread
      // per warp: 32 query rows (from q0 + 32 * quarter) against 32 key columns (from kv0)
      const int row0 = q0 + quarter * 32;
      const bool all_masked = args.causal && kv0 > row0 + 31;
      const bool need_mask = (args.causal && kv0 + 31 > row0) || (kv0 + 32 > args.Sk);
      uint32_t rs[32], rd[32];
      if (all_masked) {
        uint32_t z[16];
#pragma unroll
        for (int i = 0; i < 16; i++) z[i] = 0u;
        tmem_st16(my + 64, z);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[group]);
        continue;
      }
      tmem_ld32(my, rs);
      tmem_ld32(my + 64, rd);
      tmem_ld_wait();
      uint32_t pd[16];
      auto body = [&](auto use_mask) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
          float dv[2];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int c = 2 * i + u;
            const float e = fmaf(__uint_as_float(rs[c]), args.scale_log2, -lse2);
            float p = (HD == 64 && (c & 3) == 3 && !decltype(use_mask)::value) ? exp2_poly(e) : exp2f(e);
            if (decltype(use_mask)::value) {
              if (kv0 + c >= args.Sk || (args.causal && kv0 + c > qrow)) p = 0.f;
            }
            dv[u] = p * fmaf(__uint_as_float(rd[c]), args.scale, -dls);
          }
          pd[i] = pack16t<BF>(dv[0], dv[1]);
        }
      };
      if (need_mask) body(std::true_type{});
      else body(std::false_type{});
      tmem_st16(my + 64, pd);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[group]);
    }
    if (ok && n_sub > 0) ok = mbar_wait(acc_done, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 26);
    if (ok) {
      tc_fence_after();
      constexpr int W = HD * 4 / C::EW;
      const int cw = (group * 2 + half) * W;
      const bool row_ok = qrow < args.Sq;
      uint16_t* dqrow = (uint16_t*)args.dQ + (long long)b * args.dq_sb + (long long)qrow * args.dq_ss +
                        (long long)h * args.dq_sh + cw;
      uint32_t rr[W];
      float v[W];
      if (n_sub > 0) {
        if constexpr (W == 32) tmem_ld32(lane_addr + C::COL_ACC0 + cw, rr);
        else tmem_ld16(lane_addr + C::COL_ACC0 + cw, rr);
        tmem_ld_wait();
      }
#pragma unroll
      for (int i = 0; i < W; i++) v[i] = n_sub > 0 ? __uint_as_float(rr[i]) : 0.f;
      if (row_ok) store_row16_lim<W>(dqrow, v, BF, args.D - cw);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, C::TMEM_COLS); }
}

// dQ from the spilled dS^T: dQ[q, :] = sum over keys of dS^T[key, q] * K[key, :].  One CTA per
// 128-query tile streams 64-key slices: the dS^T slice (64 keys x 128 queries, two 64-query
// chunks) is the M-major A operand, the K slice (64 keys x HD) the N-major B operand, both
// straight from TMA-written shared memory; the accumulator is HD fp32 columns of TMEM.
// 192 threads: warp 0 TMA, warp 1 MMA, warps 2-5 the epilogue (one query row per thread).
template <int HD>
struct DqDsCfg {
  static constexpr int CH = HD / 64;
  static constexpr int DS_BYTES = 2 * BSUB * 128;        // two 64-query chunks of 64 key rows
  static constexpr int K_BYTES = CH * BSUB * 128;
  static constexpr int STAGE_BYTES = DS_BYTES + K_BYTES;
  static constexpr int NS = 4;
  static constexpr int SMEM_BYTES = NS * STAGE_BYTES + 1024 + 256;
  static constexpr int THREADS = 192;
};

template <int HD, bool BF>
__global__ void __launch_bounds__(DqDsCfg<HD>::THREADS, 2)
fa_bwd_dq_ds_kernel(const __grid_constant__ CUtensorMap tmDS, const __grid_constant__ CUtensorMap tmK,
                    const AttnArgs args) {
  using C = DqDsCfg<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = smem;
  uint64_t* bars = (uint64_t*)(ring + C::NS * C::STAGE_BYTES);
  uint64_t* full = bars;                 // NS
  uint64_t* empty = full + C::NS;        // NS
  uint64_t* acc_done = empty + C::NS;    // 1
  uint32_t* tmem_slot = (uint32_t*)(acc_done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_q_tiles = (args.Sq + BQ - 1) / BQ;
  int rank, h, b;
  block_of(args, rank, h, b);
  const int q_tile = args.causal ? num_q_tiles - 1 - rank : rank;
  const int q0 = q_tile * BQ;
  int n_sub = (args.Sk + BSUB - 1) / BSUB;
  if (args.causal) n_sub = min(n_sub, (q_tile + 1) * (BQ / BSUB));

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::NS; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(acc_done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmDS);
    tma_prefetch_desc(&tmK);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, HD); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_sub; j++) {
        if (!mbar_wait(&empty[st], ph ^ 1, abort_flag, args.status, ST_ATTN_TIMEOUT, 31)) break;
        mbar_expect_tx(&full[st], C::STAGE_BYTES);
        uint8_t* sD = ring + st * C::STAGE_BYTES;
        uint8_t* sK = sD + C::DS_BYTES;
        tma_load_4d(sD, &tmDS, &full[st], q0, j * BSUB, b * args.H + h, 0);
        tma_load_4d(sD + BSUB * 128, &tmDS, &full[st], q0 + 64, j * BSUB, b * args.H + h, 0);
#pragma unroll
        for (int c = 0; c < C::CH; c++)
          tma_load_4d(sK + c * BSUB * 128, &tmK, &full[st], c * 64, j * BSUB, h, b);
        if (++st == C::NS) { st = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc(1u, BF ? 1u : 0u, true, true, 128, HD);
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n_sub; j++) {
        if (!mbar_wait(&full[st], ph, abort_flag, args.status, ST_ATTN_TIMEOUT, 32)) break;
        tc_fence_after();
        const uint32_t da = smem_u32(ring + st * C::STAGE_BYTES), ka = da + C::DS_BYTES;
#pragma unroll
        for (int k = 0; k < BSUB / 16; k++)
          tc_mma_f16(tmem_base, mndesc_sub(da, k), mndesc_sub(ka, k), idesc, (j | k) != 0);
        tc_commit(&empty[st]);
        if (j == n_sub - 1) tc_commit(acc_done);
        if (++st == C::NS) { st = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int qrow = q0 + r;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    bool ok = true;
    if (n_sub > 0) ok = mbar_wait(acc_done, 0, abort_flag, args.status, ST_ATTN_TIMEOUT, 33);
    if (ok) {
      tc_fence_after();
      uint16_t* dqrow = (uint16_t*)args.dQ + (long long)b * args.dq_sb + (long long)qrow * args.dq_ss +
                        (long long)h * args.dq_sh;
#pragma unroll
      for (int c = 0; c < HD / 32; c++) {
        uint32_t rr[32];
        float v[32];
        if (n_sub > 0) {
          tmem_ld32(lane_addr + c * 32, rr);
          tmem_ld_wait();
        }
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = n_sub > 0 ? __uint_as_float(rr[i]) : 0.f;
        if (qrow < args.Sq) store_row16_lim<32>(dqrow + c * 32, v, BF, args.D - c * 32);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, HD); }
}

int make_qkv_map(CUtensorMap* m, const void* p, int in_bf16, int B, int H, int S, int D,
                 long long sb, long long ss, long long sh, int box_rows) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)S, (uint64_t)H, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)ss * 2, (uint64_t)sh * 2, (uint64_t)sb * 2};
  uint32_t box[4] = {64, (uint32_t)box_rows, 1, 1};
  return gbh::encode_tmap(m, in_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                          4, p, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Heads whose tiles are interleaved at the end of a causal launch: two rounds of the CTAs that run at a time.
// Measured, us in the grid's order -> so, forward and backward: (16, 12, 1024, 64) 75.4 -> 68.5, 232.7 -> 218.9; (4, 16, 2048,
// 128) 96.9 -> 81.5, 335 -> 332; (1, 16, 4096, 64) 103 -> 78, 299 -> 222; (8, 12, 600, 64) 28 -> 27, 81 -> 71; (8, 16, 4096, 128) 554 -> 534.
void fill_head_group(AttnArgs& a, int slots) {
  const long long heads = (long long)a.B * a.H, tiles = (a.Sq + BQ - 1) / BQ;
  long long g = a.causal && tiles * heads < (1LL << 31) ? (2 * slots + tiles - 1) / tiles : 0;
  if (g > heads) g = heads;
  // the products are exact while (largest dividend) * (divisor) stays below 2^32
  if (g * tiles * g >= (1LL << 32) || heads * a.H >= (1LL << 32) || a.H < 2 || g < 2) g = 0;
  a.head_group = (int)g;
  if (g == 0) return;
  a.group_recip = (unsigned)(((1ULL << 32) + g - 1) / g);
  a.head_recip = (unsigned)(((1ULL << 32) + a.H - 1) / a.H);
}

template <int HD, bool BF, int NBUF>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
               AttnArgs& a, cudaStream_t s) {
  using C = FwdCfg<HD, NBUF>;
  static bool configured = false;
  if (!configured) {
    GB_CUDA_OK(cudaFuncSetAttribute(fa_fwd_kernel<HD, BF, NBUF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    C::SMEM_BYTES));
    configured = true;
  }
  fill_head_group(a, C::CTAS_PER_SM * 148);
  dim3 grid((a.Sq + BQ - 1) / BQ, a.H, a.B);
  GB_CUDA_OK(gbh::launch(fa_fwd_kernel<HD, BF, NBUF>, grid, dim3(kFwdThreads), C::SMEM_BYTES, s, 1, tq, tk, tv, to, a));
  return gbh::E_OK;
}

struct BwdMaps {
  CUtensorMap q128, k128, v128, g128;  // 128-row boxes (resident tiles)
  CUtensorMap q64, k64, v64, g64;      // 64-row boxes (streamed sub-tiles)
  CUtensorMap dk, dv;                  // 128-row boxes
  CUtensorMap ds;                      // the dS^T spill: (query, key, batch*head), boxes of 64 x 64
  CUtensorMap ds_out;                  // the same with boxes of 64 x 128, as the dK / dV kernel writes it
};


template <int HD, bool BF>
int launch_bwd(const BwdMaps& m, const AttnArgs& a, cudaStream_t s) {
  using C = BwdCfg<HD>;
  using KV = KvCfg<HD>;
  static bool configured = false;
  if (!configured) {
    GB_CUDA_OK(cudaFuncSetAttribute(fa_bwd_dkv_kernel<HD, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, KV::SMEM_BYTES));
    GB_CUDA_OK(cudaFuncSetAttribute(fa_bwd_dq_kernel<HD, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    configured = true;
  }
  dim3 gkv((a.Sk + BKV - 1) / BKV, a.H, a.B);
  fa_bwd_dkv_kernel<HD, BF><<<gkv, KV::THREADS, KV::SMEM_BYTES, s>>>(m.q64, m.k128, m.v128, m.g64, m.ds_out, m.dk, m.dv, a);
  GB_CUDA_OK(cudaGetLastError());
  dim3 gq((a.Sq + BQ - 1) / BQ, a.H, a.B);
  if (a.dS) {
    using D = DqDsCfg<HD>;
    static bool configured_ds = false;
    if (!configured_ds) {
      GB_CUDA_OK(cudaFuncSetAttribute(fa_bwd_dq_ds_kernel<HD, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, D::SMEM_BYTES));
      configured_ds = true;
    }
    fa_bwd_dq_ds_kernel<HD, BF><<<gq, D::THREADS, D::SMEM_BYTES, s>>>(m.ds, m.k64, a);
  } else {
    fa_bwd_dq_kernel<HD, BF><<<gq, C::THREADS, C::SMEM_BYTES, s>>>(m.q128, m.k64, m.v64, m.g128, a);
  }
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

long long* g_trace = nullptr;

}  // namespace

enum { DT_BF16 = 0, DT_F16 = 1 };

// Timeline tracing of the dK/dV kernel (builds with -DGB_FA_TRACE only): `buf` is a device buffer of
// 3 * 512 int64 (zeroed by the caller) that CTA (0,0,0) fills with SM clock stamps; null switches it off.
GB_EXPORT int gb_flash_trace(long long* buf) {
  g_trace = buf;
  return 0;
}

// Forward.  q/k/v/o: 16-bit tensors addressed as [b][s][h][d] through element
// strides (sb, ss, sh) with d contiguous; head_dim a multiple of 8 up to 128.  lse (fp32,
// [B,H,Sq], natural log of the scaled scores' softmax denominator) may be null.
GB_EXPORT int gb_flash_fwd(int dtype, const void* q, const void* k, const void* v, void* o,
                           float* lse, int B, int H, int Sq, int Sk, int D, long long q_sb,
                           long long q_ss, long long q_sh, long long k_sb, long long k_ss,
                           long long k_sh, long long v_sb, long long v_ss, long long v_sh,
                           long long o_sb, long long o_ss, long long o_sh, float scale, int causal,
                           void* stream) {
  if (D < 8 || D > 128 || (D & 7)) {
    gbh::set_error("gb_flash_fwd: head_dim must be a multiple of 8 up to 128 (got %d)", D);
    return gbh::E_BAD_ARG;
  }
  if (causal && Sq != Sk) {
    gbh::set_error("gb_flash_fwd: causal attention needs Sq == Sk");
    return gbh::E_BAD_ARG;
  }
  if ((o_sb | o_ss | o_sh) & 7 || ((uintptr_t)o & 15)) {
    gbh::set_error("gb_flash_fwd: output strides must be multiples of 8 elements");
    return gbh::E_BAD_ARG;
  }
  AttnArgs a;
  memset(&a, 0, sizeof(a));
  a.B = B; a.H = H; a.Sq = Sq; a.Sk = Sk; a.D = D;
  a.scale = scale; a.scale_log2 = scale * 1.4426950408889634f;
  a.causal = causal; a.in_bf16 = dtype == DT_BF16;
  a.LSE = lse;
  a.status = gbh::status_ptr();
  CUtensorMap tq, tk, tv, to;
  int rc;
  if ((rc = make_qkv_map(&tq, q, a.in_bf16, B, H, Sq, D, q_sb, q_ss, q_sh, BQ))) return rc;
  if ((rc = make_qkv_map(&tk, k, a.in_bf16, B, H, Sk, D, k_sb, k_ss, k_sh, BKF))) return rc;
  if ((rc = make_qkv_map(&tv, v, a.in_bf16, B, H, Sk, D, v_sb, v_ss, v_sh, BKF))) return rc;
  if ((rc = make_qkv_map(&to, o, a.in_bf16, B, H, Sq, D, o_sb, o_ss, o_sh, 32))) return rc;
  // head sizes other than 64 / 128 run the next larger kernel: the tensor maps describe the real
  // extent, loads beyond it are zero-filled by TMA, stores stop at the real extent
  cudaStream_t st = (cudaStream_t)stream;
  if (D > 64) return a.in_bf16 ? launch_fwd<128, true, 2>(tq, tk, tv, to, a, st) : launch_fwd<128, false, 2>(tq, tk, tv, to, a, st);
  // Four CTAs per SM from two rounds of them on.  us, two | four CTAs per SM, heads x length: causal 768 tiles 30.8 | 31.4, 1 024 (32 x
  // 4096) 105 | 115, 1 184 (148 x 1024) 46.7 | 42.5, (74 x 2048) 72.0 | 73.1, 1 536 59.5 | 53.9, 4 096 (128 x 4096) 403 | 391;
  // not causal 768 49.5 | 50.0, 1 184 67.9 | 64.4, 2 400 135.5 | 122.6; 12 tiles of 77 5.3 | 6.4.
  const bool four = (long long)((Sq + BQ - 1) / BQ) * H * B >= 2 * FwdCfg<64, 1>::CTAS_PER_SM * 148;
  if (four) return a.in_bf16 ? launch_fwd<64, true, 1>(tq, tk, tv, to, a, st) : launch_fwd<64, false, 1>(tq, tk, tv, to, a, st);
  return a.in_bf16 ? launch_fwd<64, true, 2>(tq, tk, tv, to, a, st) : launch_fwd<64, false, 2>(tq, tk, tv, to, a, st);
}

GB_EXPORT int gb_flash_delta(int dtype, const void* o, const void* dout, float* delta, int B, int H,
                             int S, int D, long long o_sb, long long o_ss, long long o_sh,
                             long long g_sb, long long g_ss, long long g_sh, void* stream) {
  long long total = (long long)B * H * S;
  if (total < 1) return gbh::E_OK;
  const bool vec = (D == 64 || D == 128) && !((o_sb | o_ss | o_sh | g_sb | g_ss | g_sh) & 7) &&
                   !(((uintptr_t)o | (uintptr_t)dout) & 15);
  if (vec) {
    const int rows = 4 * 256 / (D / 8);         // of a CTA pass
    const int grid = (int)((total + rows - 1) / rows < 148 * 8 ? (total + rows - 1) / rows : 148 * 8);
    cudaStream_t st = (cudaStream_t)stream;
    const bool small = total < (1LL << 31) - (long long)rows * 148 * 8;      // no sum of rows overflows
#define GB_DELTA_I(T, TPR, I)                                                                             \
  fa_delta_vec_kernel<T, TPR, I><<<grid, 256, 0, st>>>((const T*)o, (const T*)dout, delta, B, H, S, o_sb, \
                                                       o_ss, o_sh, g_sb, g_ss, g_sh)
#define GB_DELTA(T, TPR)                            \
  do {                                              \
    if (small) GB_DELTA_I(T, TPR, unsigned);        \
    else GB_DELTA_I(T, TPR, long long);             \
  } while (0)
    if (dtype == DT_BF16) { if (D == 64) GB_DELTA(__nv_bfloat16, 8); else GB_DELTA(__nv_bfloat16, 16); }
    else { if (D == 64) GB_DELTA(__half, 8); else GB_DELTA(__half, 16); }
#undef GB_DELTA_I
#undef GB_DELTA
    GB_CUDA_OK(cudaGetLastError());
    return gbh::E_OK;
  }
  int grid = (int)((total + 7) / 8 < 148 * 16 ? (total + 7) / 8 : 148 * 16);
  if (dtype == DT_BF16)
    fa_delta_kernel<__nv_bfloat16><<<grid, 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, B, H, S, D, o_sb, o_ss, o_sh, g_sb, g_ss, g_sh);
  else
    fa_delta_kernel<__half><<<grid, 256, 0, (cudaStream_t)stream>>>(
        (const __half*)o, (const __half*)dout, delta, B, H, S, D, o_sb, o_ss, o_sh, g_sb, g_ss, g_sh);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// Backward.  All tensors are [b][s][h][d] through element strides, d contiguous.
// lse: the forward's output; delta: from gb_flash_delta.  Writes dq, dk, dv.
// Bytes of workspace with which gb_flash_bwd_ws computes dQ from a spilled dS^T.
GB_EXPORT long long gb_flash_bwd_ws_bytes(int B, int H, int Sq, int Sk) {
  const long long ld = (Sq + 127) / 128 * 128, rows = (Sk + 127) / 128 * 128;
  return (long long)B * H * rows * ld * 2;
}

GB_EXPORT int gb_flash_bwd_ws(int dtype, const void* q, const void* k, const void* v, const void* dout,
                              const float* lse, const float* delta, void* dq, void* dk, void* dv,
                              int B, int H, int Sq, int Sk, int D, const long long* strides,
                              float scale, int causal, void* ws, long long ws_bytes, void* stream);

GB_EXPORT int gb_flash_bwd(int dtype, const void* q, const void* k, const void* v, const void* dout,
                           const float* lse, const float* delta, void* dq, void* dk, void* dv,
                           int B, int H, int Sq, int Sk, int D, const long long* strides,
                           float scale, int causal, void* stream) {
  return gb_flash_bwd_ws(dtype, q, k, v, dout, lse, delta, dq, dk, dv, B, H, Sq, Sk, D, strides, scale, causal,
                         nullptr, 0, stream);
}

// The same with an optional workspace (32-byte aligned, gb_flash_bwd_ws_bytes bytes, contents
// arbitrary).  With it the dK/dV kernel also writes dS^T and dQ is one product dS K read back
// from it; without it (null, too small, or a problem of more than 4 GiB, the most that the caller keeps for it) a second kernel
// recomputes the scores for dQ.
GB_EXPORT int gb_flash_bwd_ws(int dtype, const void* q, const void* k, const void* v, const void* dout,
                              const float* lse, const float* delta, void* dq, void* dk, void* dv,
                              int B, int H, int Sq, int Sk, int D, const long long* strides,
                              float scale, int causal, void* ws, long long ws_bytes, void* stream) {
  // strides: 7 triples (sb, ss, sh) for q, k, v, dout, dq, dk, dv
  if (D < 8 || D > 128 || (D & 7)) {
    gbh::set_error("gb_flash_bwd: head_dim must be a multiple of 8 up to 128 (got %d)", D);
    return gbh::E_BAD_ARG;
  }
  if (causal && Sq != Sk) {
    gbh::set_error("gb_flash_bwd: causal attention needs Sq == Sk");
    return gbh::E_BAD_ARG;
  }
  for (int i = 12; i < 21; i++)
    if (strides[i] & 7) {
      gbh::set_error("gb_flash_bwd: gradient strides must be multiples of 8 elements");
      return gbh::E_BAD_ARG;
    }
  AttnArgs a;
  memset(&a, 0, sizeof(a));
  a.B = B; a.H = H; a.Sq = Sq; a.Sk = Sk; a.D = D;
  a.scale = scale; a.scale_log2 = scale * 1.4426950408889634f;
  a.causal = causal; a.in_bf16 = dtype == DT_BF16;
  fill_head_group(a, 148);
  a.LSE = const_cast<float*>(lse); a.Delta = delta;
  a.dQ = dq;
  a.dq_sb = strides[12]; a.dq_ss = strides[13]; a.dq_sh = strides[14];
  a.status = gbh::status_ptr();
  a.trace = g_trace;
  // a scale so small that LSE / scale could overflow scores like 0: the statistics are folded with 2^-100 then
  const float fold = fabsf(scale) >= 0x1p-100f ? scale : copysignf(0x1p-100f, scale);
  a.inv_scale = 1.f / fold;
  if (fold != scale) a.scale_log2 = fold * 1.4426950408889634f;
  BwdMaps m;
  memset(&m, 0, sizeof(m));
  int rc;
  if ((rc = make_qkv_map(&m.q128, q, a.in_bf16, B, H, Sq, D, strides[0], strides[1], strides[2], 128))) return rc;
  if ((rc = make_qkv_map(&m.k128, k, a.in_bf16, B, H, Sk, D, strides[3], strides[4], strides[5], 128))) return rc;
  if ((rc = make_qkv_map(&m.v128, v, a.in_bf16, B, H, Sk, D, strides[6], strides[7], strides[8], 128))) return rc;
  if ((rc = make_qkv_map(&m.g128, dout, a.in_bf16, B, H, Sq, D, strides[9], strides[10], strides[11], 128))) return rc;
  if ((rc = make_qkv_map(&m.q64, q, a.in_bf16, B, H, Sq, D, strides[0], strides[1], strides[2], 64))) return rc;
  if ((rc = make_qkv_map(&m.k64, k, a.in_bf16, B, H, Sk, D, strides[3], strides[4], strides[5], 64))) return rc;
  if ((rc = make_qkv_map(&m.v64, v, a.in_bf16, B, H, Sk, D, strides[6], strides[7], strides[8], 64))) return rc;
  if ((rc = make_qkv_map(&m.g64, dout, a.in_bf16, B, H, Sq, D, strides[9], strides[10], strides[11], 64))) return rc;
  if ((rc = make_qkv_map(&m.dk, dk, a.in_bf16, B, H, Sk, D, strides[15], strides[16], strides[17], 128))) return rc;
  if ((rc = make_qkv_map(&m.dv, dv, a.in_bf16, B, H, Sk, D, strides[18], strides[19], strides[20], 128))) return rc;
  if (ws != nullptr && ws_bytes >= gb_flash_bwd_ws_bytes(B, H, Sq, Sk) && !((uintptr_t)ws & 31) &&
      gb_flash_bwd_ws_bytes(B, H, Sq, Sk) <= (1LL << 32)) {
    a.dS = ws;
    a.ds_ld = (Sq + 127) / 128 * 128;
    a.ds_rows = (Sk + 127) / 128 * 128;
    uint64_t dims[4] = {(uint64_t)a.ds_ld, (uint64_t)a.ds_rows, (uint64_t)B * H, 1};
    uint64_t st[3] = {(uint64_t)a.ds_ld * 2, (uint64_t)a.ds_ld * a.ds_rows * 2, (uint64_t)a.ds_ld * a.ds_rows * 2 * B * H};
    uint32_t box[4] = {64, 64, 1, 1};
    if ((rc = gbh::encode_tmap(&m.ds, a.in_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                               4, ws, dims, st, box, CU_TENSOR_MAP_SWIZZLE_128B)))
      return rc;
    uint32_t box_out[3] = {64, 128, 1};
    if ((rc = gbh::encode_tmap(&m.ds_out, a.in_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                               3, ws, dims, st, box_out, CU_TENSOR_MAP_SWIZZLE_128B)))
      return rc;
  }
  if (D > 64)
    return a.in_bf16 ? launch_bwd<128, true>(m, a, (cudaStream_t)stream) : launch_bwd<128, false>(m, a, (cudaStream_t)stream);
  return a.in_bf16 ? launch_bwd<64, true>(m, a, (cudaStream_t)stream) : launch_bwd<64, false>(m, a, (cudaStream_t)stream);
}
