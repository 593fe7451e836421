// Double-precision attention on the fp64 tensor instructions (mma.sync m16n8k8 f64), head size <= 64: the
// three roles of attn_general.cu (forward, dQ, dK/dV) with the same masks, padding and dropout.
//
// What bounds it: 7 products of T x T x D forward and backward (9 where the backward recomputes dS for dQ) on a pipe of 64 fused
// multiply-adds per SM and clock (and one exponential per score and pass, 15 of them each).  The SIMT kernel
// spent its time in shared-memory reads (a 16-byte read feeds eight multiply-adds); here a fragment read of
// 16 bytes a lane feeds 32.
//  * a warp owns 16 rows (queries; keys in the dK/dV role) and its accumulators stay in registers;
//  * scores come out of the tensor instruction in the C layout (columns 2t, 2t + 1 of lane t) and are the
//    next product's A operand (columns t, t + 4) without moving: the tile row that stands at score column n
//    is chosen so that column 2t holds tile row t and column 2t + 1 tile row 4 + (t + 2) % 4, and the
//    contraction over tile rows runs in that order on both sides.  With a pitch of 4 mod 16 doubles
//    every fragment read (rows by lane group, rows by lane, both forms) is free of bank conflicts;
//  * tiles of the streamed side arrive by cp.async into two stages.
// Work split: KW warps of a CTA share 16 rows and take different rows of each tile (their sums meet in
// shared memory in a fixed order), 4 / KW row groups per CTA.  KW = 1 reuses a tile four times; small
// problems leave SMs idle that way and take KW = 2 or 4 (launch_split).
// Measured at 16 heads x 2048, D = 64, causal: forward 562 us (784 SIMT), dQ 623 (1906), dK / dV 791 (2220); the
// fp64 pipe is 57 - 70 % active (ncu), the rest is the exponentials' dependent chains, which the two
// warps per scheduler that 250 registers allow do not cover.
#include "attn_args.cuh"
#include "f64_mma.cuh"

using namespace gb;
using namespace gba;

namespace {

constexpr int kWarps = 4, kThreads = kWarps * 32;

// n rows of D columns (rows r0 .. of tensor p, batch b, head h) into a tile of pitch P; rows past `limit` and
// the columns D .. C - 1 become zero.
template <int C, int P>
__device__ __forceinline__ void issue_rows(double* dst, const void* p, const long long* s, int b, int h, int r0, int n,
                                           int limit, int D) {
  const double* base = (const double*)p + (long long)b * s[0] + (long long)h * s[2];
  const bool vec = ((reinterpret_cast<uintptr_t>(base) & 15) == 0) && (s[1] & 1) == 0 && (D & 1) == 0;
  if (vec) {
    for (int i = threadIdx.x; i < n * (C / 2); i += kThreads) {
      const int r = i / (C / 2), c = (i - r * (C / 2)) * 2;
      const bool ok = r0 + r < limit && c < D;
      cp_async16(dst + r * P + c, ok ? base + (long long)(r0 + r) * s[1] + c : base, ok ? 16 : 0);
    }
  } else {
    for (int i = threadIdx.x; i < n * C; i += kThreads) {
      const int r = i / C, c = i - r * C;
      const bool ok = r0 + r < limit && c < D;
      cp_async8(dst + r * P + c, ok ? base + (long long)(r0 + r) * s[1] + c : base, ok ? 8 : 0);
    }
  }
}

template <int MODE, int DT, int KW, int NT>
struct Shape {
  static constexpr int C = DT * 8;              // columns held (D rounded up)
  static constexpr int P = C + 4;               // pitch: 4 mod 16 for C = 16, 32, 64
  static constexpr int RW = kWarps / KW;        // row groups
  static constexpr int ROWS = RW * 16;
  static constexpr int TK = KW * NT * 8;        // tile rows
  static constexpr int ROW_BUFS = MODE == MODE_FWD ? 1 : 2;
  static constexpr int STAGE = 2 * TK * P + (MODE == MODE_DKV ? 2 * TK : 0);
  static constexpr int DOUBLES = ROW_BUFS * ROWS * P + 2 * STAGE;
  static constexpr int BYTES = DOUBLES * 8;
  // the partial sums of the KW warps of a row group meet in the tile buffers
  static constexpr int OUTS = MODE == MODE_DKV ? 2 : 1;
  static_assert(KW == 1 || kWarps * 16 * P + 2 * kWarps * 16 <= DOUBLES, "merge buffer");
};

template <int MODE, int DT, int KW, int NT>
__global__ void __launch_bounds__(kThreads, 2) attn_f64_kernel(const GArgs a) {
  using S = Shape<MODE, DT, KW, NT>;
  constexpr int P = S::P, TK = S::TK, ROWS = S::ROWS;
  extern __shared__ __align__(16) double fsm[];
  double* rowsA = fsm;                                   // FWD / DQ: Q; DKV: K
  double* rowsB = rowsA + ROWS * P;                      // DQ: dO; DKV: V
  double* stages = rowsA + S::ROW_BUFS * ROWS * P;       // two of: tile A (K; DKV: Q), tile B (V; DKV: dO), lse, delta
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wk = warp % KW, wr = warp / KW;              // slice of each tile, row group
  const int yt = 4 + ((t + 2) & 3);                      // tile row at score column 2t + 1
  const int gp = (g & 1) ? 4 + (((g >> 1) + 2) & 3) : (g >> 1);   // tile row at score column g
  const int nrows = MODE == MODE_DKV ? a.Tk : a.Tq, ntile = MODE == MODE_DKV ? a.Tq : a.Tk;
  const bool pure_causal = a.causal && a.mask == nullptr && a.kpm == nullptr;
  // All heads' blocks of one row range start together; causal blocks differ in length, the longest go
  // first (in the grid's own order the last head's longest block ended the kernel: 772 against 562 us
  // forward at 16 heads of 2048).
  const long long lin = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
  const long long heads = (long long)gridDim.y * gridDim.z;
  const int rank = (int)(lin / heads), bh = (int)(lin - rank * heads), b = bh / a.H, h = bh - b * a.H;
  const int bx = (MODE != MODE_DKV && pure_causal) ? (int)gridDim.x - 1 - rank : rank;
  const int row0 = bx * ROWS;
  const int wrow = row0 + wr * 16;                       // the warp's first row
  const uint32_t thresh = (uint32_t)fmin(a.p_drop * 4294967296.0, 4294967295.0);
  const double keep_scale = a.p_drop > 0.0 ? 1.0 / (1.0 - a.p_drop) : 1.0;
  const double* LSEp = reinterpret_cast<const double*>(a.LSE) + (long long)bh * a.Tq;
  const double* Deltap = reinterpret_cast<const double*>(a.Delta) + (long long)bh * a.Tq;

  int t_begin = 0, t_end = ntile;                        // pure causal attention never looks past the diagonal
  if (pure_causal) {
    if (MODE == MODE_DKV) t_begin = row0 / TK * TK;
    else t_end = min(ntile, row0 + ROWS);
  }
  auto issue = [&](int st, int t0) {
    double* ta = stages + st * S::STAGE;
    if (t0 < t_end) {
      if (MODE == MODE_DKV) {
        issue_rows<S::C, P>(ta, a.Q, a.q_s, b, h, t0, TK, a.Tq, a.D);
        issue_rows<S::C, P>(ta + TK * P, a.dO, a.g_s, b, h, t0, TK, a.Tq, a.D);
        double* ls = ta + 2 * TK * P;
        for (int i = threadIdx.x; i < 2 * TK; i += kThreads) {
          const int q = t0 + (i < TK ? i : i - TK);
          const double* src = i < TK ? LSEp : Deltap;
          cp_async8(ls + i, q < a.Tq ? src + q : src, q < a.Tq ? 8 : 0);
        }
      } else {
        issue_rows<S::C, P>(ta, a.K, a.k_s, b, h, t0, TK, a.Tk, a.D);
        issue_rows<S::C, P>(ta + TK * P, a.V, a.v_s, b, h, t0, TK, a.Tk, a.D);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (MODE == MODE_DKV) {
    issue_rows<S::C, P>(rowsA, a.K, a.k_s, b, h, row0, ROWS, a.Tk, a.D);
    issue_rows<S::C, P>(rowsB, a.V, a.v_s, b, h, row0, ROWS, a.Tk, a.D);
  } else {
    issue_rows<S::C, P>(rowsA, a.Q, a.q_s, b, h, row0, ROWS, a.Tq, a.D);
    if (MODE == MODE_DQ) issue_rows<S::C, P>(rowsB, a.dO, a.g_s, b, h, row0, ROWS, a.Tq, a.D);
  }
  issue(0, t_begin);

  double acc[DT][4], acc2[MODE == MODE_DKV ? DT : 1][4];
#pragma unroll
  for (int n = 0; n < DT; n++)
#pragma unroll
    for (int e = 0; e < 4; e++) {
      acc[n][e] = 0.0;
      if (MODE == MODE_DKV) acc2[n][e] = 0.0;
    }
  double m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0, 0.0};   // FWD: running maximum, this lane's part of the sum
  double lse_r[2] = {0.0, 0.0}, delta_r[2] = {0.0, 0.0};
  if (MODE == MODE_DQ) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int row = wrow + g + 8 * r;
      if (row < a.Tq) { lse_r[r] = LSEp[row]; delta_r[r] = Deltap[row]; }
    }
  }
  double qf[MODE == MODE_FWD ? DT : 1][4];                   // FWD: the query rows as A fragments
  const double* arow = rowsA + (wr * 16 + g) * P + t;
  const double* brow = rowsB + (wr * 16 + g) * P + t;

  for (int t0 = t_begin, st = 0; t0 < t_end; t0 += TK, st ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                         // tile t0 is there, the other stage is no longer read
    issue(st ^ 1, t0 + TK);
    if (MODE == MODE_FWD && t0 == t_begin) {
#pragma unroll
      for (int k = 0; k < DT; k++) {
        qf[k][0] = arow[k * 8]; qf[k][1] = arow[8 * P + k * 8];
        qf[k][2] = arow[k * 8 + 4]; qf[k][3] = arow[8 * P + k * 8 + 4];
      }
    }
    const int u0 = t0 + wk * (NT * 8);                       // the warp's first tile row
    if (u0 >= ntile) continue;
    if (pure_causal && (MODE == MODE_DKV ? u0 + NT * 8 - 1 < wrow : u0 > wrow + 15)) continue;   // exact zeros
    const double* ta = stages + st * S::STAGE + wk * (NT * 8) * P;
    const double* tb = ta + TK * P;
    // ---- scores (and dO V^T) of 16 rows against NT * 8 tile rows ----
    double s[NT][4], dp[MODE == MODE_FWD ? 1 : NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        s[j][e] = 0.0;
        if (MODE != MODE_FWD) dp[j][e] = 0.0;
      }
#pragma unroll
    for (int k = 0; k < DT; k++) {
      double a0, a1, a2, a3;
      if (MODE == MODE_FWD) {
        a0 = qf[k][0]; a1 = qf[k][1]; a2 = qf[k][2]; a3 = qf[k][3];
      } else {
        a0 = arow[k * 8]; a1 = arow[8 * P + k * 8]; a2 = arow[k * 8 + 4]; a3 = arow[8 * P + k * 8 + 4];
      }
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const double* x = ta + (j * 8 + gp) * P + k * 8 + t;
        dmma(s[j], a0, a1, a2, a3, x[0], x[4]);
      }
      if (MODE != MODE_FWD) {
        const double d0 = brow[k * 8], d1 = brow[8 * P + k * 8], d2 = brow[k * 8 + 4], d3 = brow[8 * P + k * 8 + 4];
#pragma unroll
        for (int j = 0; j < NT; j++) {
          const double* x = tb + (j * 8 + gp) * P + k * 8 + t;
          dmma(dp[j], d0, d1, d2, d3, x[0], x[4]);
        }
      }
    }
    // ---- masks and softmax terms ----
    double mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int row = wrow + g + 8 * (e >> 1), col = u0 + j * 8 + ((e & 1) ? yt : t);
        const int qi = MODE == MODE_DKV ? col : row, ki = MODE == MODE_DKV ? row : col;
        double v = s[j][e] * a.scale;
        if (row < nrows && col < ntile) {
          if (a.causal && ki > qi) v += -1e30;
          if (a.mask) v += (double)a.mask[(long long)qi * a.Tk + ki];
          if (a.kpm && a.kpm[(long long)b * a.Tk + ki]) v += -1e30;
        }
        if (col >= ntile) v = -INFINITY;                     // takes no part
        s[j][e] = v;
        if (MODE == MODE_FWD) mx[e >> 1] = fmax(mx[e >> 1], v);
      }
    if (MODE == MODE_FWD) {
      bool moved = false;
      double corr[2];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        mx[r] = fmax(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
        mx[r] = fmax(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
        const double mn = fmax(m[r], mx[r]);
        corr[r] = m[r] == mn ? 1.0 : exp(m[r] - mn);         // m = -inf: 0
        moved |= m[r] != mn;
        m[r] = mn;
      }
      if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
        for (int r = 0; r < 2; r++) l[r] *= corr[r];
#pragma unroll
        for (int n = 0; n < DT; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[n][e] *= corr[e >> 1];
      }
    }
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int row = wrow + g + 8 * (e >> 1), col = u0 + j * 8 + ((e & 1) ? yt : t);
        const int qi = MODE == MODE_DKV ? col : row, ki = MODE == MODE_DKV ? row : col;
        const bool valid = row < nrows && col < ntile;
        const bool keep = !(a.p_drop > 0.0) || !valid || keep_cell(a, bh, qi, ki, thresh);
        if (MODE == MODE_FWD) {
          // a row whose scores are all -inf so far has no weights yet
          const double p = m[e >> 1] == -INFINITY ? 0.0 : exp(s[j][e] - m[e >> 1]);
          l[e >> 1] += p;
          s[j][e] = keep ? p * keep_scale : 0.0;
        } else {
          const double* ls = stages + st * S::STAGE + 2 * TK * P;
          const int ci = wk * (NT * 8) + j * 8 + ((e & 1) ? yt : t);
          const double lse = MODE == MODE_DKV ? ls[ci] : lse_r[e >> 1];
          const double delta = MODE == MODE_DKV ? ls[TK + ci] : delta_r[e >> 1];
          const double p = valid ? exp(s[j][e] - lse) : 0.0;
          const double dpd = keep ? dp[j][e] * keep_scale : 0.0;
          s[j][e] = p * (dpd - delta) * a.scale;
          dp[j][e] = keep ? p * keep_scale : 0.0;
          if (MODE == MODE_DKV && a.dS != nullptr && valid) a.dS[((long long)bh * a.ds_rows + row) * a.ds_ld + col] = s[j][e];
        }
      }
    // ---- FWD: acc += p V   DQ: acc += ds K   DKV: acc += ds Q, acc2 += p' dO ----
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const double* x = (MODE == MODE_FWD ? tb : ta) + j * 8 * P + g;
#pragma unroll
      for (int n = 0; n < DT; n++) dmma(acc[n], s[j][0], s[j][2], s[j][1], s[j][3], x[t * P + n * 8], x[yt * P + n * 8]);
      if (MODE == MODE_DKV) {
        const double* y = tb + j * 8 * P + g;
#pragma unroll
        for (int n = 0; n < DT; n++) dmma(acc2[n], dp[j][0], dp[j][2], dp[j][1], dp[j][3], y[t * P + n * 8], y[yt * P + n * 8]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");

  if (MODE == MODE_FWD) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
  }
  auto out_row = [&](int which, int row) {
    void* p = MODE == MODE_FWD ? a.O : MODE == MODE_DQ ? a.dQ : which == 0 ? a.dK : a.dV;
    const long long* st = MODE == MODE_FWD ? a.o_s : MODE == MODE_DQ ? a.dq_s : which == 0 ? a.dk_s : a.dv_s;
    return (double*)p + (long long)b * st[0] + (long long)row * st[1] + (long long)h * st[2];
  };
  if (KW == 1) {
    double inv[2] = {1.0, 1.0};
    if (MODE == MODE_FWD) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        inv[r] = 1.0 / l[r];                                 // l = 0 (every score -inf): 0 * inf, not a number
        const int row = wrow + g + 8 * r;
        if (t == 0 && row < nrows && a.LSE)
          const_cast<double*>(LSEp)[row] = l[r] > 0.0 ? m[r] + log(l[r]) : -INFINITY;
      }
    }
#pragma unroll
    for (int which = 0; which < S::OUTS; which++)
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int row = wrow + g + 8 * r;
        if (row >= nrows) continue;
        double* o = out_row(which, row);
#pragma unroll
        for (int n = 0; n < DT; n++)
#pragma unroll
          for (int e = 0; e < 2; e++)
            if (n * 8 + 2 * t + e < a.D) o[n * 8 + 2 * t + e] = (which == 0 ? acc[n] : acc2[n])[2 * r + e] * inv[r];
      }
    return;
  }
  // ---- KW > 1: the warps of a row group add up in warp order ----
  double* part = fsm;                                        // [kWarps][16][P]
  double* ml = fsm + kWarps * 16 * P;                        // FWD: [kWarps][16] maxima, [kWarps][16] sums
#pragma unroll
  for (int which = 0; which < S::OUTS; which++) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
      double* d = part + (warp * 16 + g + 8 * r) * P + 2 * t;
#pragma unroll
      for (int n = 0; n < DT; n++)
#pragma unroll
        for (int e = 0; e < 2; e++) d[n * 8 + e] = (which == 0 ? acc[n] : acc2[n])[2 * r + e];
      if (MODE == MODE_FWD && t == 0) {
        ml[warp * 16 + g + 8 * r] = m[r];
        ml[(kWarps + warp) * 16 + g + 8 * r] = l[r];
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ROWS * S::C; i += kThreads) {
      const int rr = i / S::C, c = i - rr * S::C, w0 = rr / 16 * KW, r16 = rr % 16;
      const int row = row0 + rr;
      if (row >= nrows || c >= a.D) continue;
      double v = 0.0;
      if (MODE == MODE_FWD) {
        double mm = -INFINITY, ll = 0.0;
#pragma unroll
        for (int w = 0; w < KW; w++) mm = fmax(mm, ml[(w0 + w) * 16 + r16]);
#pragma unroll
        for (int w = 0; w < KW; w++) {
          const double mw = ml[(w0 + w) * 16 + r16];
          const double f = mw == -INFINITY ? 0.0 : exp(mw - mm);
          ll += f * ml[(kWarps + w0 + w) * 16 + r16];
          v += f * part[((w0 + w) * 16 + r16) * P + c];
        }
        v *= 1.0 / ll;
        if (c == 0 && a.LSE) const_cast<double*>(LSEp)[row] = ll > 0.0 ? mm + log(ll) : -INFINITY;
      } else {
#pragma unroll
        for (int w = 0; w < KW; w++) v += part[((w0 + w) * 16 + r16) * P + c];
      }
      out_row(which, row)[c] = v;
    }
  }
}

// dQ = dS K from the dS^T that the dK / dV role left in memory: one product instead of three and the exponentials.  A
// warp owns 16 queries; tiles of 32 keys, [key][query] and [key][column], pitch 4 mod 16: conflict-free fragments.
// Bound by the fp64 pipe and the read of dS^T (268 MB at 16 heads of 2048, causal: backward 1438 -> 1024 us).
template <int DT>
struct DqShape {
  static constexpr int C = DT * 8, P = C + 4, ROWS = 64, PS = ROWS + 4, TK = 32;
  static constexpr int STAGE = TK * (P + PS), BYTES = 2 * STAGE * 8;
};
template <int DT>
__global__ void __launch_bounds__(kThreads, 3) attn_f64_dq_ds_kernel(const GArgs a) {
  using S = DqShape<DT>;
  constexpr int P = S::P, PS = S::PS, TK = S::TK;
  extern __shared__ __align__(16) double fsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool pure_causal = a.causal && a.mask == nullptr && a.kpm == nullptr;
  const long long lin = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
  const long long heads = (long long)gridDim.y * gridDim.z;
  const int rank = (int)(lin / heads), bh = (int)(lin - rank * heads), b = bh / a.H, h = bh - b * a.H;
  const int row0 = (pure_causal ? (int)gridDim.x - 1 - rank : rank) * S::ROWS;      // longest first
  const int t_end = pure_causal ? min(a.Tk, row0 + S::ROWS) : a.Tk;
  const double* ds = a.dS + (long long)bh * a.ds_rows * a.ds_ld + row0;
  auto issue = [&](int st, int t0) {
    if (t0 < t_end) {
      double* ts = fsm + st * S::STAGE;
      for (int i = threadIdx.x; i < TK * (S::ROWS / 2); i += kThreads) {      // rows of dS^T are 64-padded and aligned
        const int r = i / (S::ROWS / 2), c = (i - r * (S::ROWS / 2)) * 2;
        const bool ok = t0 + r < a.Tk;
        cp_async16(ts + r * PS + c, ok ? ds + (long long)(t0 + r) * a.ds_ld + c : ds, ok ? 16 : 0);
      }
      issue_rows<S::C, P>(ts + TK * PS, a.K, a.k_s, b, h, t0, TK, a.Tk, a.D);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[DT][4];
#pragma unroll
  for (int n = 0; n < DT; n++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[n][e] = 0.0;
  issue(0, 0);
  const int q = row0 + warp * 16 + g;
  for (int t0 = 0, st = 0; t0 < t_end; t0 += TK, st ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    issue(st ^ 1, t0 + TK);
    const double* ts = fsm + st * S::STAGE + t * PS + warp * 16 + g;
    const double* tk = fsm + st * S::STAGE + TK * PS + t * P + g;
    // above the diagonal of pure causal attention nothing was written (queries past Tq: never written either, their rows of
    // dQ are not stored)
    const bool diagonal = pure_causal && t0 + TK - 1 > row0 + warp * 16;
#pragma unroll
    for (int k = 0; k < TK; k += 8) {
      double a0 = ts[k * PS], a1 = ts[k * PS + 8], a2 = ts[(k + 4) * PS], a3 = ts[(k + 4) * PS + 8];
      if (diagonal) {
        const int key = t0 + k + t;
        a0 = key > q ? 0.0 : a0;
        a1 = key > q + 8 ? 0.0 : a1;
        a2 = key + 4 > q ? 0.0 : a2;
        a3 = key + 4 > q + 8 ? 0.0 : a3;
      }
#pragma unroll
      for (int n = 0; n < DT; n++) dmma(acc[n], a0, a1, a2, a3, tk[k * P + n * 8], tk[(k + 4) * P + n * 8]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int r = 0; r < 2; r++) {
    if (q + 8 * r >= a.Tq) continue;
    double* o = (double*)a.dQ + (long long)b * a.dq_s[0] + (long long)(q + 8 * r) * a.dq_s[1] + (long long)h * a.dq_s[2];
#pragma unroll
    for (int n = 0; n < DT; n++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        if (n * 8 + 2 * t + e < a.D) o[n * 8 + 2 * t + e] = acc[n][2 * r + e];
  }
}

template <int DT>
int launch_dq_ds(const GArgs& a, cudaStream_t s) {
  auto k = attn_f64_dq_ds_kernel<DT>;
  GB_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, DqShape<DT>::BYTES));
  k<<<dim3((a.Tq + 63) / 64, a.H, a.B), kThreads, DqShape<DT>::BYTES, s>>>(a);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

int g_f64_split = 0;      // 0: by the rule below; 1, 2, 4: that many warps per row group

template <int MODE, int DT, int KW, int NT>
int launch_one(const GArgs& a, cudaStream_t s) {
  using S = Shape<MODE, DT, KW, NT>;
  auto k = attn_f64_kernel<MODE, DT, KW, NT>;
  GB_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES));
  const int rows = MODE == MODE_DKV ? a.Tk : a.Tq;
  k<<<dim3((rows + S::ROWS - 1) / S::ROWS, a.H, a.B), kThreads, S::BYTES, s>>>(a);
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// How many warps share a row group.  Measured, us forward / dQ / dK and dV, KW = 1 | 2 | 4:
//   16 heads x 2048, D = 64, causal (512 blocks of 64 rows)   562/651/812 | 598/623/791 | 767/735/898
//   16 x 2048, D = 16 (512)                                   646/623/736 | 569/530/788 | 698/561/735
//   16 x 1200, D = 32, causal (304)                           248/251/285 | 162/148/183 | 222/164/233
//   8 x 1024, D = 64 (128)                                    241/256/322 | 177/182/233 | 223/211/256
//   8 x 1024, D = 64, causal (128)                            239/256/322 | 159/159/202 | 113/106/128
//   8 x 512, D = 64 (64)                                      123/133/166 |  80/ 75/ 94 |  66/ 59/ 71
// and for full GPUs, forward / dK and dV, KW = 1 | 2:
//   8 x 512 x 16, causal (1024) 310/461 | 364/450     4 x 1024 x 16 (1024) 1133/1748 | 1198/1661
//   2 x 2048 x 16, causal (1024) 1050/1612 | 1165/1578    1 x 2048 x 16 (512) 1138/1798 | 1284/1832
// KW = 1 needs 1.5 waves of two CTAs per SM and the long accumulation of wide heads to pay for its coarse
// blocks, and pays in the forward alone, whose row state (running maximum and sum) every merge has to bring
// together; KW = 4 pays while KW = 2 leaves SMs without a second CTA (causal blocks are half as long on average).
template <int MODE, int DT>
int launch_split(const GArgs& a, cudaStream_t s) {
  const int rows = MODE == MODE_DKV ? a.Tk : a.Tq;
  const long long blocks64 = (long long)((rows + 63) / 64) * a.H * a.B;
  const int kw = g_f64_split ? g_f64_split
                             : MODE == MODE_FWD && blocks64 >= 444 && a.D > 32 ? 1 : blocks64 >= (a.causal ? 200 : 100) ? 2 : 4;
  if (kw == 1) return launch_one<MODE, DT, 1, MODE == MODE_FWD ? 4 : 2>(a, s);   // 104 KB: two CTAs per SM
  if (kw == 2) return launch_one<MODE, DT, 2, 2>(a, s);
  return launch_one<MODE, DT, 4, 1>(a, s);
}

template <int MODE>
int launch_mode(const GArgs& a, cudaStream_t s) {
  if (a.D <= 16) return launch_split<MODE, 2>(a, s);
  if (a.D <= 32) return launch_split<MODE, 4>(a, s);
  return launch_split<MODE, 8>(a, s);
}

}  // namespace

int gba::launch_f64(int mode, const GArgs& a, cudaStream_t s) {
  if (mode == MODE_FWD) return launch_mode<MODE_FWD>(a, s);
  if (mode == MODE_DQ && a.dS != nullptr)
    return a.D <= 16 ? launch_dq_ds<2>(a, s) : a.D <= 32 ? launch_dq_ds<4>(a, s) : launch_dq_ds<8>(a, s);
  if (mode == MODE_DQ) return launch_mode<MODE_DQ>(a, s);
  return launch_mode<MODE_DKV>(a, s);
}

// Warps that share a row group in the fp64 kernels: 1, 2 or 4, 0 = chosen by size (for measurements and tests).
GB_EXPORT int gb_attn_f64_tune(int split) {
  if (split != 0 && split != 1 && split != 2 && split != 4) {
    gbh::set_error("gb_attn_f64_tune: split is 0, 1, 2 or 4");
    return gbh::E_BAD_ARG;
  }
  g_f64_split = split;
  return gbh::E_OK;
}
