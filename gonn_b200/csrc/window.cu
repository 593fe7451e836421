// Sliding-window core shared by convolution, pooling, fold / unfold and padding.
//
// The reference builds, for every sliding-window layer, a dense 0/1 "gather
// matrix" G (numWin*winSize x prod(In)) and applies it with a GEMM
// (nn/gather.go:99-181, nn/conv.go:341-380, nn/pool.go:340-370).  Here the same
// information is an int32 index map idx[win][tap] (-1 = padding) and the gather
// is done by address: no multiply by zeros, no dense matrix.  The transpose of
// the gather (col2im, pooling backward) uses the inverted map in CSR form, so it
// is a gather too: deterministic, no atomics.
//
//   window_gather   col[n][win][c*T + tap] = x[n][c][idx[win][tap]]   (im2col; the row
//                   of one window is K-major for the GEMM that follows)
//   window_scatter  dx[n][c][i] = sum over (win,tap) with idx[win][tap]==i of
//                   dcol[n][win][c*T + tap]                              (col2im)
//   pool_fwd / pool_bwd   max (with argmax), average, LP-norm pooling over idx
#include "bounds.cuh"

using namespace gb;

namespace {

// q = i / d, r = i % d; 32-bit arithmetic when both operands fit (64-bit division costs
// tens of instructions and these kernels do one or two per element).
__device__ __forceinline__ void divmod(long long i, long long d, bool small, long long& q, long long& r) {
  if (small) {
    const unsigned ii = (unsigned)i, dd = (unsigned)d;
    const unsigned qq = ii / dd;
    q = qq;
    r = ii - qq * dd;
  } else {
    q = i / d;
    r = i - q * d;
  }
}

template <typename T>
__global__ void window_gather_kernel(const T* __restrict__ x, const int* __restrict__ idx,
                                     T* __restrict__ col, int N, int C, long long S, int nwin, int T_,
                                     int kpad, float fill) {
  // one thread per (n, win, k) with k = c*T + tap; k in [0, kpad), zero beyond C*T
  const long long total = (long long)N * nwin * kpad;
  const bool small = total <= 0x7fffffffLL;
  const int K = C * T_;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long r, kk, nn, ww;
    divmod(i, kpad, small, r, kk);
    divmod(r, nwin, small, nn, ww);
    const int k = (int)kk, win = (int)ww, n = (int)nn;
    T v = (T)0.f;
    if (k < K) {
      const int c = k / T_, tap = k - c * T_;
      const int src = idx[win * T_ + tap];
      v = (src >= 0 && GB_IN_BOUNDS(src, S, 101)) ? x[((long long)n * C + c) * S + src] : (T)fill;
    }
    col[i] = v;
  }
}

// dx[n][c][i] = sum_{e in csr(i)} dcol[n][win(e)][c*T + tap(e)], csr_cols[e] = win*T + tap
template <typename T>
__global__ void window_scatter_kernel(const T* __restrict__ dcol, const int* __restrict__ offs,
                                      const int* __restrict__ cols, T* __restrict__ dx, int N, int C,
                                      long long S, int nwin, int T_, int kpad, int accumulate) {
  const long long total = (long long)N * C * S;
  const bool small = total <= 0x7fffffffLL;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long pos, r, cc, nn;
    divmod(i, S, small, r, pos);
    divmod(r, C, small, nn, cc);
    const int c = (int)cc, n = (int)nn;
    float acc = 0.f;
    for (int e = offs[pos]; e < offs[pos + 1]; e++) {
      const int wt = cols[e];
      const int win = wt / T_, tap = wt - win * T_;
      if (!GB_IN_BOUNDS(wt, (long long)nwin * T_, 102)) continue;
      acc += (float)dcol[((long long)n * nwin + win) * kpad + c * T_ + tap];
    }
    dx[i] = accumulate ? (T)((float)dx[i] + acc) : (T)acc;
  }
}

enum PoolMode : int { POOL_MAX = 0, POOL_AVG = 1, POOL_LP = 2 };

// y[b][win] over taps idx[win][*]; b = n*C + c.  arg[b][win] = winning tap (max).
template <typename T>
__global__ void pool_fwd_kernel(const T* __restrict__ x, const int* __restrict__ idx,
                                T* __restrict__ y, int* __restrict__ arg, long long B, long long S,
                                int nwin, int T_, int mode, int count_include_pad, float p) {
  pdl_trigger();
  pdl_wait();
  const long long total = B * nwin;
  const bool small = total <= 0x7fffffffLL && B * S <= 0x7fffffffLL;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long b, ww;
    divmod(i, nwin, small, b, ww);
    const int win = (int)ww;
    const T* xb = x + b * S;
    const int* iw = idx + (long long)win * T_;
    if (mode == POOL_MAX) {
      float best = -INFINITY;
      int bt = -1;
      for (int t = 0; t < T_; t++) {
        const int src = iw[t];
        if (src < 0 || !GB_IN_BOUNDS(src, S, 103)) continue;
        const float v = (float)xb[src];
        if (v > best || bt < 0) { best = v; bt = t; }
      }
      y[i] = (T)(bt < 0 ? 0.f : best);
      if (arg) arg[i] = bt;
    } else if (mode == POOL_AVG) {
      float s = 0.f;
      int cnt = 0;
      for (int t = 0; t < T_; t++) {
        const int src = iw[t];
        if (src >= 0 && GB_IN_BOUNDS(src, S, 104)) { s += (float)xb[src]; cnt++; }
      }
      const int div = count_include_pad ? T_ : (cnt > 0 ? cnt : 1);
      y[i] = (T)(s / (float)div);
    } else {
      float s = 0.f;
      for (int t = 0; t < T_; t++) {
        const int src = iw[t];
        if (src >= 0 && GB_IN_BOUNDS(src, S, 105)) s += powf((float)xb[src], p);
      }
      y[i] = (T)powf(s, 1.f / p);
    }
  }
}

// Max / average pooling with at most TAPS = 4 or 8 taps per window (2 x 2, 2 x 2 x 2, ...): a thread keeps the
// tap offsets of its windows in registers and walks the planes of its blockIdx.y slice, U at a time so that their loads are in
// flight together.  What bounds it is instructions (130 a window with eight tested taps, 16384 x 900 bf16 28 us; now 12.5): a tap
// that is padding reads the first one that is not again, which neither wins a maximum nor counts in a sum, so the loop tests
// nothing.
template <typename T, int TAPS, bool MAX>
__global__ void __launch_bounds__(256)
pool_fwd_small_kernel(const T* __restrict__ x, const int* __restrict__ idx, T* __restrict__ y, int* __restrict__ arg, long long B,
                      long long S, int nwin, int T_, int count_include_pad) {
  pdl_trigger();
  pdl_wait();
  constexpr int U = 16 / TAPS;
  for (int win = blockIdx.x * blockDim.x + threadIdx.x; win < nwin; win += gridDim.x * blockDim.x) {
    int src[TAPS], first = -1, cnt = 0;
    unsigned valid = 0;
#pragma unroll
    for (int t = 0; t < TAPS; t++) {
      src[t] = t < T_ ? __ldg(idx + (long long)win * T_ + t) : -1;
      if (src[t] >= 0 && !GB_IN_BOUNDS(src[t], S, 108)) src[t] = -1;
      if (src[t] >= 0) {
        valid |= 1u << t;
        cnt++;
        if (first < 0) first = t;
      }
    }
    int pad = 0;
#pragma unroll
    for (int t = 0; t < TAPS; t++) pad = t == first ? src[t] : pad;
#pragma unroll
    for (int t = 0; t < TAPS; t++) src[t] = src[t] < 0 ? pad : src[t];
    const float inv = 1.f / (float)(count_include_pad ? T_ : (cnt > 0 ? cnt : 1));
    const T* xb = x + (long long)blockIdx.y * S;
    long long o = (long long)blockIdx.y * nwin + win;
    const long long x_step = (long long)gridDim.y * S, o_step = (long long)gridDim.y * nwin;
    auto one = [&](const float (&v)[TAPS], long long at) {
      if (MAX) {
        float best = v[0];
        int bt = first;
#pragma unroll
        for (int t = 1; t < TAPS; t++) {
          const bool more = v[t] > best;
          best = more ? v[t] : best;
          bt = more ? t : bt;
        }
        y[at] = (T)(first < 0 ? 0.f : best);
        if (arg) arg[at] = bt;
      } else {
        float sum = 0.f;
#pragma unroll
        for (int t = 0; t < TAPS; t++) sum += valid >> t & 1u ? v[t] : 0.f;
        y[at] = (T)(sum * inv);
      }
    };
    long long b = blockIdx.y;
    for (; b + (U - 1) * (long long)gridDim.y < B; b += (long long)gridDim.y * U) {
      float v[U][TAPS];
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int t = 0; t < TAPS; t++) v[u][t] = (float)xb[u * x_step + src[t]];
#pragma unroll
      for (int u = 0; u < U; u++) one(v[u], o + u * o_step);
      xb += U * x_step;
      o += U * o_step;
    }
    for (; b < B; b += gridDim.y) {
      float v[TAPS];
#pragma unroll
      for (int t = 0; t < TAPS; t++) v[t] = (float)xb[src[t]];
      one(v, o);
      xb += x_step;
      o += o_step;
    }
  }
}

// Max / average pooling over wide windows (global pooling: one window of H * W taps): one warp per
// output, lanes along the taps, then a shuffle reduction.  The arg-max is the first tap that holds the
// maximum, as in the one-thread-per-output kernel.
template <typename T>
__global__ void pool_fwd_wide_kernel(const T* __restrict__ x, const int* __restrict__ idx, T* __restrict__ y,
                                     int* __restrict__ arg, long long B, long long S, int nwin, int T_, int mode,
                                     int count_include_pad) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const long long total = B * nwin;
  for (long long o = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); o < total; o += (long long)gridDim.x * wpb) {
    const long long b = o / nwin;
    const int win = (int)(o - b * nwin);
    const T* xb = x + b * S;
    const int* iw = idx + (long long)win * T_;
    float best = -INFINITY, sum = 0.f;
    int bt = 0x7fffffff, cnt = 0;
    for (int t = lane; t < T_; t += 32) {
      const int src = __ldg(iw + t);
      if (src < 0 || !GB_IN_BOUNDS(src, S, 109)) continue;
      const float v = (float)xb[src];
      sum += v;
      cnt++;
      if (v > best || bt == 0x7fffffff) { best = v; bt = t; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, off);
      const int ot = __shfl_xor_sync(0xffffffffu, bt, off);
      sum += __shfl_xor_sync(0xffffffffu, sum, off);
      cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
      // a lane that saw no tap holds (-inf, INT_MAX) and always loses; equal values keep the earlier tap
      if (ot != 0x7fffffff && (bt == 0x7fffffff || ov > best || (ov == best && ot < bt))) { best = ov; bt = ot; }
    }
    if (lane == 0) {
      if (mode == POOL_MAX) {
        y[o] = (T)(bt == 0x7fffffff ? 0.f : best);
        if (arg) arg[o] = bt == 0x7fffffff ? -1 : bt;
      } else {
        y[o] = (T)(sum / (float)(count_include_pad ? T_ : (cnt > 0 ? cnt : 1)));
      }
    }
  }
}

// The same for windows of at most 32 NT taps where there are many planes: a warp stays with one window, keeps the taps' offsets in
// registers and has the loads of U planes in flight together (a maximum one plane's: its selections are what a warp waits for, and
// with more planes fewer warps fit).
template <typename T, int NT, bool MAX>
__global__ void __launch_bounds__(256)
pool_fwd_stay_kernel(const T* __restrict__ x, const int* __restrict__ idx, T* __restrict__ y, int* __restrict__ arg, long long B,
                     long long S, int nwin, int T_, int count_include_pad) {
  pdl_trigger();
  pdl_wait();
  constexpr int U = MAX ? 1 : 16 / NT;
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const long long warps = (long long)gridDim.x * wpb, w0 = (long long)blockIdx.x * wpb + (threadIdx.x >> 5);
  const long long per = warps / nwin;            // warps of a window (the launch has at least one each)
  if (w0 >= per * nwin) return;
  const int win = (int)(w0 % nwin);
  int off[NT], cnt = 0;
#pragma unroll
  for (int k = 0; k < NT; k++) {
    const int t = lane + 32 * k;
    off[k] = t < T_ ? __ldg(idx + (long long)win * T_ + t) : -1;
    if (off[k] >= 0 && !GB_IN_BOUNDS(off[k], S, 109)) off[k] = -1;
    cnt += off[k] >= 0;
  }
  float div = (float)T_;
  if (!MAX && !count_include_pad) {
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    div = (float)(cnt > 0 ? cnt : 1);
  }
  for (long long b = w0 / nwin; b < B; b += per * U) {
    float v[U][NT];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const T* xb = x + (b + u * per) * S;
#pragma unroll
      for (int k = 0; k < NT; k++) v[u][k] = off[k] >= 0 && b + u * per < B ? (float)xb[off[k]] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (b + u * per >= B) break;               // (the same for the whole warp)
      const long long o = (b + u * per) * nwin + win;
      if (MAX) {
        float best = -INFINITY;
        int bt = 0x7fffffff;
#pragma unroll
        for (int k = 0; k < NT; k++)
          if (off[k] >= 0 && (v[u][k] > best || bt == 0x7fffffff)) { best = v[u][k]; bt = lane + 32 * k; }
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, best, q);
          const int ot = __shfl_xor_sync(0xffffffffu, bt, q);
          if (ot != 0x7fffffff && (bt == 0x7fffffff || ov > best || (ov == best && ot < bt))) { best = ov; bt = ot; }
        }
        if (lane == 0) {
          y[o] = (T)(bt == 0x7fffffff ? 0.f : best);
          if (arg) arg[o] = bt == 0x7fffffff ? -1 : bt;
        }
      } else {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < NT; k++) sum += v[u][k];
        sum = warp_sum(sum);
        if (lane == 0) y[o] = (T)(sum / div);
      }
    }
  }
}

// dx[b][i] = sum over (win,tap) covering i of the window's gradient share
template <typename T>
__global__ void pool_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                const T* __restrict__ y, const int* __restrict__ arg,
                                const int* __restrict__ idx, const int* __restrict__ offs,
                                const int* __restrict__ cols, T* __restrict__ dx, long long B,
                                long long S, int nwin, int T_, int mode, int count_include_pad,
                                float p) {
  pdl_trigger();
  pdl_wait();
  const long long total = B * S;
  const bool small = total <= 0x7fffffffLL;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long pos, b;
    divmod(i, S, small, b, pos);
    float acc = 0.f;
    for (int e = offs[pos]; e < offs[pos + 1]; e++) {
      const int wt = cols[e];
      const int win = wt / T_, tap = wt - win * T_;
      if (!GB_IN_BOUNDS(wt, (long long)nwin * T_, 106)) continue;
      const long long o = b * nwin + win;
      if (mode == POOL_MAX) {
        if (arg[o] == tap) acc += (float)dy[o];
      } else if (mode == POOL_AVG) {
        int div = T_;
        if (!count_include_pad) {
          int cnt = 0;
          for (int t = 0; t < T_; t++) cnt += idx[(long long)win * T_ + t] >= 0;
          div = cnt > 0 ? cnt : 1;
        }
        acc += (float)dy[o] / (float)div;
      } else {
        // d/dx (sum x^p)^(1/p) = x^(p-1) * y^(1-p)
        const float yv = (float)y[o];
        if (yv != 0.f) acc += (float)dy[o] * powf((float)x[i], p - 1.f) * powf(yv, 1.f - p);
      }
    }
    dx[i] = (T)acc;
  }
}

// Backward of max / average pooling whose windows do not overlap (every input position lies in at
// most one window: the usual stride == kernel case and global pooling).  p2w[pos] = {window, tap}
// of the position, or {-1, 0}; wcnt[win] = taps of the window that are not padding.  One thread
// per input element, rows (b) along blockIdx.y: no division, one table read and two dependent
// loads per element, coalesced stores.
template <typename T, bool MAX>
__global__ void __launch_bounds__(256)
pool_bwd_disjoint_kernel(const T* __restrict__ dy, const int* __restrict__ arg, const int2* __restrict__ p2w, const int* __restrict__ wcnt,
                         T* __restrict__ dx, long long B, int S, int nwin, int T_, int count_include_pad) {
  pdl_trigger();
  pdl_wait();
  // A thread keeps its positions' table entries in registers and walks the planes (b) of its blockIdx.y slice, U at a time so that
  // their loads are in flight together (a position outside every window reads window 0 and stores 0).  16384 x 900, 2 x 2 windows,
  // bf16: four at a time 31 us, so 19.9.
  constexpr int U = 8;
  for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < S; pos += gridDim.x * blockDim.x) {
    const int2 w = __ldg(p2w + pos);
    const bool hit = w.x >= 0 && GB_IN_BOUNDS(w.x, nwin, 107);
    const int win = hit ? w.x : 0, tap = hit ? w.y : -2;      // (no arg-max is -2)
    float inv = 0.f;
    if (hit && !MAX) inv = 1.f / (float)(count_include_pad ? T_ : max(__ldg(wcnt + w.x), 1));
    long long b = blockIdx.y, o = (long long)blockIdx.y * nwin + win, i = (long long)blockIdx.y * S + pos;
    const long long step = gridDim.y, o_step = step * nwin, i_step = step * S;
    for (; b + (U - 1) * step < B; b += U * step) {
      float g[U];
      int a[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        g[u] = (float)dy[o + u * o_step];
        if (MAX) a[u] = arg[o + u * o_step];
      }
#pragma unroll
      for (int u = 0; u < U; u++) dx[i + u * i_step] = (T)(MAX ? (a[u] == tap ? g[u] : 0.f) : hit ? g[u] * inv : 0.f);
      o += U * o_step;
      i += U * i_step;
    }
    for (; b < B; b += step) {
      const float g = (float)dy[o];
      dx[i] = (T)(MAX ? (arg[o] == tap ? g : 0.f) : hit ? g * inv : 0.f);
      o += o_step;
      i += i_step;
    }
  }
}

inline int grid_for(long long work) {
  long long g = (work + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

enum { DT_BF16 = 0, DT_F16 = 1, DT_F32 = 2, DT_F64 = 3 };

#define GB_DISPATCH_T(CALL)                                   \
  switch (dtype) {                                            \
    case DT_BF16: { using T = __nv_bfloat16; CALL; } break;   \
    case DT_F16: { using T = __half; CALL; } break;           \
    case DT_F32: { using T = float; CALL; } break;            \
    default:                                                  \
      gbh::set_error("window op: unsupported dtype %d", dtype); \
      return gbh::E_BAD_ARG;                                  \
  }

// im2col: x (N,C,S) -> col (N, nwin, kpad) with K = C*T real columns (zero padded to kpad)
GB_EXPORT int gb_window_gather(int dtype, const void* x, const int* idx, void* col, int N, int C,
                               long long S, int nwin, int T_, int kpad, float fill, void* stream) {
  const long long total = (long long)N * nwin * kpad;
  if (total <= 0) return gbh::E_OK;
  cudaStream_t s = (cudaStream_t)stream;
  GB_BOUNDS_BIND();
  GB_DISPATCH_T((window_gather_kernel<T><<<grid_for(total), 256, 0, s>>>((const T*)x, idx, (T*)col, N, C, S, nwin, T_, kpad, fill)));
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// col2im: dcol (N, nwin, kpad) -> dx (N,C,S) through the inverted index map (CSR over S)
GB_EXPORT int gb_window_scatter(int dtype, const void* dcol, const int* offs, const int* cols,
                                void* dx, int N, int C, long long S, int nwin, int T_, int kpad,
                                int accumulate, void* stream) {
  const long long total = (long long)N * C * S;
  if (total <= 0) return gbh::E_OK;
  cudaStream_t s = (cudaStream_t)stream;
  GB_BOUNDS_BIND();
  GB_DISPATCH_T((window_scatter_kernel<T><<<grid_for(total), 256, 0, s>>>((const T*)dcol, offs, cols, (T*)dx, N, C, S, nwin, T_, kpad, accumulate)));
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// mode: 0 max (arg receives the winning tap per window, may be null), 1 average, 2 LP norm
GB_EXPORT int gb_pool_fwd(int dtype, const void* x, const int* idx, void* y, int* arg, long long B,
                          long long S, int nwin, int T_, int mode, int count_include_pad, float p,
                          void* stream) {
  const long long total = B * nwin;
  if (total <= 0) return gbh::E_OK;
  cudaStream_t s = (cudaStream_t)stream;
  GB_BOUNDS_BIND();
  // (an empty plane under padding alone has no element that a tap of padding could read again)
  if (mode != POOL_LP && T_ <= 8 && B >= 64 && S > 0) {
    const int bx = (nwin + 255) / 256 < 64 ? (nwin + 255) / 256 : 64;
    long long by = (148 * 8 + bx - 1) / bx;
    if (by > B) by = B;
#define GB_POOL(TAPS, MAX) gbh::launch(pool_fwd_small_kernel<T, TAPS, MAX>, dim3(dim3(bx, (unsigned)by)), dim3(256), 0, s, 1, (const T*)x, idx, (T*)y, arg, B, S, nwin, T_, count_include_pad)
    GB_DISPATCH_T(({
      if (T_ <= 4) { if (mode == POOL_MAX) GB_POOL(4, true); else GB_POOL(4, false); }
      else { if (mode == POOL_MAX) GB_POOL(8, true); else GB_POOL(8, false); }
    }));
#undef GB_POOL
    GB_CUDA_OK(cudaGetLastError());
    return gbh::E_OK;
  }
  if (mode != POOL_LP && T_ >= 64) {
    const long long most = 148 * 8;
    const unsigned grid = (unsigned)((total + 7) / 8 < most ? (total + 7) / 8 : most);
    // Staying pays where a warp has several planes of its window (bf16, us, walking | staying: average over 64 taps, 8 192 outputs 10.2 |
    // 10.4, 32 768 18.3 | 12.4, 1.2 M 424 | 184; maximum over 169 taps, 2 048 outputs 8.3 | 10.1, 8 192 10.4 | 10.2, 295 K 139 | 100), and
    // where the warps divide among the windows (6 400 windows of 64 taps on 64 planes 548 | 566).  More than 256 taps would not stay
    // in registers: 1 024 taps on 8 192 planes 22 | 37, 3 136 on 2 048 29 | 56 with the rest read behind them.
    const int nt = (T_ + 31) / 32;
    const bool stay = T_ <= 256 && nwin * 4ll <= grid * 8ll && total >= (mode == POOL_MAX ? 4096 : 16384);
#define GB_STAY_(NT, MAX) gbh::launch(pool_fwd_stay_kernel<T, NT, MAX>, dim3(grid), dim3(256), 0, s, 1, (const T*)x, idx, (T*)y, arg, B, S, nwin, T_, count_include_pad)
#define GB_STAY(NT) { if (mode == POOL_MAX) GB_STAY_(NT, true); else GB_STAY_(NT, false); }
    GB_DISPATCH_T(({
      if (!stay) gbh::launch(pool_fwd_wide_kernel<T>, dim3(grid), dim3(256), 0, s, 1, (const T*)x, idx, (T*)y, arg, B, S, nwin, T_, mode, count_include_pad);
      else if (nt <= 2) GB_STAY(2)
      else if (nt == 3) GB_STAY(3)
      else if (nt == 4) GB_STAY(4)
      else if (nt == 5) GB_STAY(5)
      else if (nt == 6) GB_STAY(6)
      else if (nt == 7) GB_STAY(7)
      else GB_STAY(8)
    }));
#undef GB_STAY
#undef GB_STAY_
    GB_CUDA_OK(cudaGetLastError());
    return gbh::E_OK;
  }
  GB_DISPATCH_T((gbh::launch(pool_fwd_kernel<T>, dim3(grid_for(total)), dim3(256), 0, s, 1, (const T*)x, idx, (T*)y, arg, B, S, nwin, T_, mode, count_include_pad, p)));
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

// Backward for non-overlapping windows (max or average): see pool_bwd_disjoint_kernel.
GB_EXPORT int gb_pool_bwd_disjoint(int dtype, const void* dy, const int* arg, const int* p2w, const int* wcnt,
                                   void* dx, long long B, long long S, int nwin, int T_, int mode,
                                   int count_include_pad, void* stream) {
  if (B <= 0 || S <= 0) return gbh::E_OK;
  if (mode != POOL_MAX && mode != POOL_AVG) {
    gbh::set_error("gb_pool_bwd_disjoint: max or average pooling only");
    return gbh::E_BAD_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  GB_BOUNDS_BIND();
  const int bx = (int)((S + 255) / 256 < 64 ? (S + 255) / 256 : 64);
  // about eight CTAs per SM in total; every CTA walks B / by planes
  long long by = (148 * 8 + bx - 1) / bx;
  if (by > B) by = B;
  if (by < 1) by = 1;
  GB_DISPATCH_T(({
    if (mode == POOL_MAX) gbh::launch(pool_bwd_disjoint_kernel<T, true>, dim3(dim3(bx, (unsigned)by)), dim3(256), 0, s, 1, (const T*)dy, arg, (const int2*)p2w, wcnt, (T*)dx, B, (int)S, nwin, T_, count_include_pad);
    else gbh::launch(pool_bwd_disjoint_kernel<T, false>, dim3(dim3(bx, (unsigned)by)), dim3(256), 0, s, 1, (const T*)dy, arg, (const int2*)p2w, wcnt, (T*)dx, B, (int)S, nwin, T_, count_include_pad);
  }));
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}

GB_EXPORT int gb_pool_bwd(int dtype, const void* dy, const void* x, const void* y, const int* arg,
                          const int* idx, const int* offs, const int* cols, void* dx, long long B,
                          long long S, int nwin, int T_, int mode, int count_include_pad, float p,
                          void* stream) {
  const long long total = B * S;
  if (total <= 0) return gbh::E_OK;
  cudaStream_t s = (cudaStream_t)stream;
  GB_BOUNDS_BIND();
  GB_DISPATCH_T((gbh::launch(pool_bwd_kernel<T>, dim3(grid_for(total)), dim3(256), 0, s, 1, (const T*)dy, (const T*)x, (const T*)y, arg, idx, offs, cols, (T*)dx, B, S, nwin, T_, mode, count_include_pad, p)));
  GB_CUDA_OK(cudaGetLastError());
  return gbh::E_OK;
}
