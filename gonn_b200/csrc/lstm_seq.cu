// A whole LSTM layer over a batch of sequences in one persistent kernel per direction (fp32).
//
// The recurrence is a chain of T products of B x H by H x 4H that no larger GEMM can replace: what
// bounds it is the latency of one step, not arithmetic (B = 32, H = 512: 33.5 M multiply-adds, 0.9 us
// of the FMA pipes).  Launched step by step (one small GEMM, one gate kernel and the tape's additions
// per step) a step costs 70 us forward and 270 us with its backward, most of it launches and a GEMM
// that fills 16 SMs.  Here
//  * the recurrent weight stays in shared memory for the whole sequence: a CTA owns UT hidden units
//    (their four gate rows forward, their column of W_hh backward) for a group of sequences;
//  * sequences are independent, so only the CTAs of one group wait for one another.  Forward: h_t travels as 64-bit
//    words {value, step + 1} in a buffer of two steps by turns; a reader loads the words it needs and repeats those whose
//    step is not there yet, so that no flag, fence or second round trip stands between a product and the next (a flag
//    per CTA with release semantics: 6.3 us a step).  A warp receives the part of h that its share of the contraction needs
//    and starts on it at once (4.2 -> 3.8 us against a barrier behind the whole of h).  A word of step t is overwritten by
//    step t + 2, whose writer has read step t + 1 from every CTA of its group, and each of those had read step t before.
//    Backward: the sums of dh_t travel the same way (lstm_seq_bwd_scatter_kernel); where their words would take too much
//    memory, dgates_t are gathered (four times the data) behind H / UT flags per group, one per CTA, stored with release
//    semantics after the CTA's part of dgates_t is written, all polled by one warp;
//  * within a CTA the eight warps split the contraction, a lane accumulates 4 x 4 outputs with packed
//    fp32 multiply-adds, and the partial sums meet in shared memory in a fixed order (deterministic);
//  * the cell state never leaves the thread that owns it except to be saved for the backward.
// The input projections of all steps, the weight gradients and the input gradient are single
// GEMMs outside (ops/rnn.py).  Measured at B = 32, T = 64, H = 512: 244 us forward (3.8 us a step, 1.1 of it the multiply-adds)
// and 256 us backward (4.0); at H = 64 a step is 2.0 and 1.5 us, which is the exchange alone.
//
// Waiting CTAs need one another to be resident: cooperative launches only.  Every wait is bounded.
#include "common.cuh"

using namespace gb;

namespace {

constexpr int kMB = 8;        // sequences of one sub-tile
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

__device__ __forceinline__ float sigm(float x) { return 1.f / (1.f + __expf(-x)); }

// acc (two packed floats) += a * b
__device__ __forceinline__ void ffma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct SeqArgs {
  int B, T, H;
  int sub;                    // sub-tiles of kMB sequences per CTA
  int ug;                     // CTAs per group (hidden-unit slices)
  const float* w;             // W_hh (4H, H)
  const float* h0;            // (B, H) or null
  const float* c0;            // (B, H) or null
  unsigned int* flags;        // [groups][ug], zeroed before the launch
  int* status;
  // forward
  float* xg;                  // (B, T, 4H): x W_ih^T; with a tape replaced by the activated gates i, f, g, o
  const float* bias;          // (4H) or null
  float* out;                 // (B, T, H): h_t; without a tape sequences out_sb elements apart
  long long out_sb;
  float* hprev;               // tape: (B, T, H): h_{t-1}, for the gradient of W_hh
  float* cseq;                // tape: (B, T, H): c_t; without one (B, H): the cell state, replaced in every step
  unsigned long long* xch;    // [2][B][H] words of the exchange, zeroed before the launch
  // backward (reads cseq, (B, T, H), and act)
  const float* act;           // (B, T, 4H): activated gates
  const float* dout;          // (B, T, H) or null
  const float* dcn;           // (B, H) or null: gradient of the last cell state
  float* dgates;              // (B, T, 4H)
  float* dc0;                 // (B, H) or null
};

// Publishes this CTA's step (`value` steps done).  Called after a __syncthreads that follows the stores.
__device__ __forceinline__ void publish(unsigned int* flag, unsigned int value) {
  if (threadIdx.x == 0)
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(value) : "memory");
}

// All threads wait until every CTA of the group has published `value`; false when the budget ran out.
__device__ __forceinline__ bool wait_group(const unsigned int* flags, int n, unsigned int value, int* abort_flag,
                                           int* status) {
  if (threadIdx.x < 32) {
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    for (;;) {
      bool ok = true;
      for (int i = (int)threadIdx.x; i < n; i += 32) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + i) : "memory");
        ok = ok && v >= value;
      }
      if (__all_sync(0xffffffffu, ok)) break;
      if ((++spins & 0xFF) == 0 && globaltimer_ns() - t0 > kWaitBudgetNs) {
        if (threadIdx.x == 0) {
          *abort_flag = 1;
          set_status(status, ST_RNN_TIMEOUT, (int)value);
        }
        break;
      }
    }
  }
  __syncthreads();
  return *(volatile int*)abort_flag == 0;
}

// a: kMB rows, w: N rows, both K floats with pitch K + 4 (16-byte rows four banks apart, so that the
// 16-byte reads of eight neighbouring rows touch all banks once).  Lanes: two groups of four a-rows
// x N/4 groups of w-rows (w row = i * N/4 + group: neighbouring lanes, neighbouring rows) x KQ
// slices of the warp's share of the contraction: every kWarps-th step of it, or (OWN) its part k0 .. k1.  part[warp][kMB * N]
// receives the warp's partial sums.
template <int N, bool OWN>
__device__ __forceinline__ void product(const float* __restrict__ a, const float* __restrict__ w, int K, int k0, int k1,
                                        float* __restrict__ part) {
  constexpr int NG = N / 4;                  // groups of w-rows
  constexpr int KQ = 32 / (2 * NG);          // lanes that share a group pair and split k
  static_assert(KQ >= 1, "N <= 64");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kq = lane % KQ, ng = (lane / KQ) % NG, mg = lane / (KQ * NG);
  const int pitch = K + 4;
  const float* ap = a + (mg * 4) * pitch;
  const float* wp = w + ng * pitch;
  unsigned long long acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
#pragma unroll 2
  for (int k = OWN ? k0 + kq * 4 : (warp * KQ + kq) * 4; k < (OWN ? k1 : K); k += (OWN ? 1 : kWarps) * KQ * 4) {
    ulonglong2 av[4], wv[4];
#pragma unroll
    for (int i = 0; i < 4; i++) av[i] = *reinterpret_cast<const ulonglong2*>(ap + i * pitch + k);
#pragma unroll
    for (int j = 0; j < 4; j++) wv[j] = *reinterpret_cast<const ulonglong2*>(wp + j * NG * pitch + k);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        ffma2(acc[i][j], av[i].x, wv[j].x);
        ffma2(acc[i][j], av[i].y, wv[j].y);
      }
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float v = __uint_as_float((unsigned)(acc[i][j] & 0xffffffffull)) + __uint_as_float((unsigned)(acc[i][j] >> 32));
#pragma unroll
      for (int o = 1; o < KQ; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (kq == 0) part[warp * (kMB * N) + (mg * 4 + i) * N + j * NG + ng] = v;
    }
}

// Rows b0 .. b0 + kMB - 1 of src (row stride `stride`, K floats each) into the tile; rows past B are zero.
__device__ __forceinline__ void load_tile(float* __restrict__ tile, const float* __restrict__ src, long long stride, int K,
                                          int b0, int B) {
  const int k4 = K / 4, pitch = K + 4;
  for (int i = threadIdx.x; i < kMB * k4; i += kThreads) {
    const int r = i / k4, c = (i - r * k4) * 4;
    float* d = tile + r * pitch + c;
    if (src != nullptr && b0 + r < B)
      cp_async16(d, src + (long long)(b0 + r) * stride + c, 16);
    else
      *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  cp_async_wait_all();
}

// The part k0 .. k1 (multiples of four) of h of the step whose words carry `step` (its index + 1), rows b0 .. b0 + kMB - 1, into the
// tile, by one warp, which alone reads it: no barrier stands between the words and its product, and no warp waits for words of
// another's part.  OWN = false: k0 .. k1 by all threads of the CTA, a barrier follows (and the places of the words are worked out
// again where they are needed: kept in registers, 64 x 64 steps at H = 720 take 1 190 us instead of 1 142).  Rows past B are zero.
// Gives up when the budget of the wait has run out for any thread of the CTA.
template <bool OWN>
__device__ __forceinline__ void receive_part(float* __restrict__ tile, const unsigned long long* __restrict__ xch, unsigned step, int H,
                                             int k0, int k1, int b0, int B, int* abort_flag, int* status) {
  constexpr int U = 8;
  constexpr int W = OWN ? 32 : kThreads;
  const int h2 = (k1 - k0) / 2, pitch = H + 4, total = kMB * h2;
  for (int i0 = OWN ? threadIdx.x & 31 : threadIdx.x; i0 < total; i0 += W * U) {
    unsigned long long w[U][2];
    int at[OWN ? U : 1];
    auto place = [&](int u) {                      // row << 16 | column
      const int i = i0 + u * W, r = i / h2;
      return r << 16 | (k0 + 2 * (i - r * h2));
    };
    unsigned todo = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int to = place(u);
      if (OWN) at[u] = to;
      if (i0 + u * W < total && b0 + (to >> 16) < B) todo |= 1u << u;
    }
    const unsigned mine = todo;
    uint64_t t0 = 0;
    for (uint32_t spins = 0; todo != 0; spins++) {
#pragma unroll
      for (int u = 0; u < U; u++)
        if (todo >> u & 1u) {
          const int from = OWN ? at[u] : place(u);
          const unsigned long long* src = xch + (long long)(b0 + (from >> 16)) * H + (from & 0xffff);
          asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w[u][0]), "=l"(w[u][1]) : "l"(src) : "memory");
        }
#pragma unroll
      for (int u = 0; u < U; u++)
        if ((unsigned)(w[u][0] >> 32) == step && (unsigned)(w[u][1] >> 32) == step) todo &= ~(1u << u);
      if (todo != 0 && (spins & 0xFF) == 0xFF) {
        if (t0 == 0) t0 = globaltimer_ns();
        if (*(volatile int*)abort_flag) break;
        if (globaltimer_ns() - t0 > kWaitBudgetNs) {
          *(volatile int*)abort_flag = 1;
          set_status(status, ST_RNN_TIMEOUT, (int)step);
          break;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + u * W < total) {
        const float2 v = mine >> u & 1u ? make_float2(__uint_as_float((unsigned)w[u][0]), __uint_as_float((unsigned)w[u][1]))
                                        : make_float2(0.f, 0.f);
        const int to = OWN ? at[u] : place(u);
        *reinterpret_cast<float2*>(tile + (to >> 16) * pitch + (to & 0xffff)) = v;
      }
  }
  __syncwarp();
}

// grid: (ug, groups).  UT units per CTA: N = 4 UT weight rows, row n = gate * UT + unit.  TAPE: a backward follows (a template
// parameter and the stores in this order: with strides and flags at run time a step takes 0.2 us longer).  PARTS: buffers of partial
// sums.  With two a warp may be a product ahead of the cells; where the weights leave room for one (16 units, H from 692 to 744), a
// barrier stands before each product instead of half the units a CTA and, for many sequences, three times the dependent
// exchanges.  64 steps, us, 8 units and two buffers | 16 units and one:
// B = 64, H = 720 2 443 | 1 142, 256, 720 9 790 | 4 185, 64, 692 2 143 | 1 347, 64, 744 2 441 | 1 158.
template <int UT, bool TAPE, int PARTS>
__global__ void __launch_bounds__(kThreads, 1) lstm_seq_fwd_kernel(const SeqArgs p) {
  constexpr int N = 4 * UT;
  extern __shared__ __align__(16) float sm[];
  __shared__ int abort_flag;
  const int H = p.H, T = p.T, pitch = H + 4;
  float* ws = sm;                                  // [N][H + 4]
  float* hs = ws + N * pitch;                      // [kMB][H + 4]
  float* parts = hs + kMB * pitch;                 // [PARTS][kWarps][kMB * N], by turns
  const int u0 = blockIdx.x * UT;
  const int bg0 = blockIdx.y * p.sub * kMB;
  if (threadIdx.x == 0) abort_flag = 0;
  for (int i = threadIdx.x; i < N * (H / 4); i += kThreads) {
    const int n = i / (H / 4), c = (i - n * (H / 4)) * 4;
    const int g = n / UT, u = u0 + (n - g * UT);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (u < H) v = *reinterpret_cast<const float4*>(p.w + ((long long)g * H + u) * H + c);
    *reinterpret_cast<float4*>(ws + n * pitch + c) = v;
  }
  __syncthreads();
  const int cell_m = threadIdx.x / UT, cell_u = threadIdx.x % UT;      // the cell of threads 0 .. kMB * UT - 1
  const int u = u0 + cell_u;
  const bool cell = threadIdx.x < kMB * UT && u < H;
  const int kper = (H / 4 + kWarps - 1) / kWarps * 4, k0 = min(H, (int)(threadIdx.x >> 5) * kper), k1 = min(H, k0 + kper);   // of this warp
  float bias[4] = {0.f, 0.f, 0.f, 0.f};
  if (cell && p.bias != nullptr) {
#pragma unroll
    for (int g = 0; g < 4; g++) bias[g] = p.bias[g * H + u];
  }
  int turn = 0;
  for (int t = 0; t < T; t++) {
    for (int s = 0; s < p.sub; s++) {
      float* part = parts + (turn = (turn + 1) % PARTS) * (kWarps * kMB * N);
      const int b0 = bg0 + s * kMB, b = b0 + cell_m;
      const bool mine = cell && b < p.B;
      const long long row = (long long)b * T + t;
      float pre[4] = {0.f, 0.f, 0.f, 0.f}, cp = 0.f;
      if (mine) {                                  // in flight during the product
#pragma unroll
        for (int g = 0; g < 4; g++) pre[g] = p.xg[row * 4 * H + g * H + u] + bias[g];   // (not __ldg: this thread writes there)
        cp = t > 0 ? p.cseq[(TAPE ? row - 1 : (long long)b) * H + u] : (p.c0 != nullptr ? p.c0[(long long)b * H + u] : 0.f);
      }
      if (t > 0 || p.h0 != nullptr) {
        if (t > 0) {
          receive_part<PARTS == 2>(hs, p.xch + (long long)((t - 1) & 1) * p.B * H, (unsigned)t, H, PARTS == 2 ? k0 : 0, PARTS == 2 ? k1 : H, b0,
                                   p.B, &abort_flag, p.status);
        } else {
          load_tile(hs, p.h0, H, H, b0, p.B);
          __syncthreads();
        }
        if (PARTS == 1) __syncthreads();           // the cells have read the sums of the product before; h is whole
        product<N, PARTS == 2>(hs, ws, H, k0, k1, part);
        __syncthreads();
        if (*(volatile int*)&abort_flag != 0) return;
        if (mine) {
#pragma unroll
          for (int g = 0; g < 4; g++) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; w++) v += part[w * (kMB * N) + cell_m * N + g * UT + cell_u];
            pre[g] += v;
          }
        }
      }
      if (mine) {
        const float ig = sigm(pre[0]), fg = sigm(pre[1]), gg = tanhf(pre[2]), og = sigm(pre[3]);
        const float cn = fg * cp + ig * gg;
        const float h = og * tanhf(cn);
        if (t + 1 < T)        // first: the others wait for it
          asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p.xch + ((long long)(t & 1) * p.B + b) * H + u),
                       "l"((unsigned long long)__float_as_uint(h) | (unsigned long long)(t + 1) << 32)
                       : "memory");
        p.out[(TAPE ? row * H : b * p.out_sb + (long long)t * H) + u] = h;
        p.cseq[(TAPE ? row : (long long)b) * H + u] = cn;
        if (TAPE) {
          float* a = p.xg + row * 4 * H + u;
          a[0] = ig; a[H] = fg; a[2 * H] = gg; a[3 * H] = og;
          if (t + 1 < T) p.hprev[(row + 1) * H + u] = h;
          if (t == 0) p.hprev[row * H + u] = p.h0 != nullptr ? p.h0[(long long)b * H + u] : 0.f;
        }
      }
    }
  }
}

// grid: (ug, groups).  UT units per CTA: N = UT columns of W_hh, contraction over the 4H gates.
// (A warp takes every eighth step of the contraction: with a connected part each, 64 steps at B = 256, H = 720 take 11 620 us instead
// of 11 040.)
template <int UT>
__global__ void __launch_bounds__(kThreads, 1) lstm_seq_bwd_kernel(const SeqArgs p) {
  constexpr int N = UT;
  extern __shared__ __align__(16) float sm[];
  __shared__ int abort_flag;
  const int H = p.H, T = p.T, K = 4 * H, pitch = K + 4;
  float* ws = sm;                                  // [N][4H + 4]: column u of W_hh
  float* ds = ws + N * pitch;                      // [kMB][4H + 4]: dgates_{t+1}
  float* part = ds + kMB * pitch;                  // [kWarps][kMB * N]
  float* dcs = part + kWarps * kMB * N;            // [sub][kMB * N]: dc carried from step to step
  const int u0 = blockIdx.x * UT;
  const int bg0 = blockIdx.y * p.sub * kMB;
  unsigned int* flags = p.flags + (long long)blockIdx.y * p.ug;
  if (threadIdx.x == 0) abort_flag = 0;
  for (int i = threadIdx.x; i < N * K; i += kThreads) {
    const int n = i % UT, k = i / UT;
    ws[n * pitch + k] = u0 + n < H ? p.w[(long long)k * H + u0 + n] : 0.f;
  }
  const int cell_m = threadIdx.x / UT, cell_u = threadIdx.x % UT;
  const int u = u0 + cell_u;
  const bool cell = threadIdx.x < kMB * UT && u < H;
  for (int s = 0; s < p.sub; s++) {
    const int b = bg0 + s * kMB + cell_m;
    if (threadIdx.x < kMB * UT)
      dcs[s * (kMB * N) + threadIdx.x] = (cell && b < p.B && p.dcn != nullptr) ? p.dcn[(long long)b * H + u] : 0.f;
  }
  __syncthreads();
  for (int t = T - 1; t >= 0; t--) {
    const bool chain = t < T - 1;
    if (chain && !wait_group(flags, p.ug, (unsigned)(T - 1 - t), &abort_flag, p.status)) return;
    for (int s = 0; s < p.sub; s++) {
      const int b0 = bg0 + s * kMB, b = b0 + cell_m;
      const bool mine = cell && b < p.B;
      const long long row = (long long)b * T + t;
      float dh = 0.f, ig = 0.f, fg = 0.f, gg = 0.f, og = 0.f, ct = 0.f, cp = 0.f;
      if (mine) {
        const float* a = p.act + row * K + u;
        ig = __ldg(a); fg = __ldg(a + H); gg = __ldg(a + 2 * H); og = __ldg(a + 3 * H);
        ct = __ldg(p.cseq + row * H + u);
        cp = t > 0 ? __ldg(p.cseq + (row - 1) * H + u) : (p.c0 != nullptr ? p.c0[(long long)b * H + u] : 0.f);
        if (p.dout != nullptr) dh = __ldg(p.dout + row * H + u);
      }
      if (chain) {
        load_tile(ds, p.dgates + (long long)(t + 1) * K, (long long)T * K, K, b0, p.B);
        __syncthreads();
        product<N, false>(ds, ws, K, 0, K, part);
        __syncthreads();
        if (mine) {
          float v = 0.f;
#pragma unroll
          for (int w = 0; w < kWarps; w++) v += part[w * (kMB * N) + cell_m * N + cell_u];
          dh += v;
        }
      }
      if (mine) {
        const float tc = tanhf(ct);
        float* dcv = dcs + s * (kMB * N) + threadIdx.x;
        const float dc = *dcv + dh * og * (1.f - tc * tc);
        float* d = p.dgates + row * K + u;
        d[0] = dc * gg * ig * (1.f - ig);
        d[H] = dc * cp * fg * (1.f - fg);
        d[2 * H] = dc * ig * (1.f - gg * gg);
        d[3 * H] = dh * tc * og * (1.f - og);
        *dcv = dc * fg;
        if (t == 0 && p.dc0 != nullptr) p.dc0[(long long)b * H + u] = dc * fg;
      }
    }
    __syncthreads();
    publish(flags + blockIdx.x, (unsigned)(T - t));
  }
}

// The same chain with the exchange turned round.  The kernel above gathers all of dgates_{t+1} (4H values a sequence) in every CTA.
// Here a CTA multiplies only the dgates of its own UT units, by the 4 UT rows of W_hh that belong to them, and sends every other
// CTA the UT sums of dh_t that it owns: H values a sequence and CTA instead of 4H, in 64-bit words {value, step} as forward, so
// that neither a flag nor a second round trip stands between two steps.  A CTA adds what the others sent in their order.  Slots
// go by turns: a word of step t is overwritten by step t - 2, whose writer has the sums of step t - 1 from every CTA of its
// group, and each of those had added up step t before it sent them.
// us a step of 64, gathered | scattered: B = 32, H = 512 7.3 | 4.0; 32, 128 3.3 | 1.7; 4, 64 2.4 | 1.5; 8, 256 3.8 | 1.9;
// 128, 512 24.8 | 14.4; 512, 512 86.8 | 64.2.
// U: words in flight per thread, the senders of a cell that one thread adds up (16 at H = 512: 278 -> 256 us for 64 steps; more
// than there are costs 5 %).  grid: (ug, groups).  Words: [slot][sub-tile][receiver][sender][kMB * UT].
template <int UT, int U>
__global__ void __launch_bounds__(kThreads, 1) lstm_seq_bwd_scatter_kernel(const SeqArgs p) {
  constexpr int K = 4 * UT, pitch = K + 4, CELLS = kMB * UT;
  constexpr int PARTS = kThreads / CELLS;          // threads that share the senders of one cell
  extern __shared__ __align__(16) float sm[];
  __shared__ int abort_flag;
  const int H = p.H, T = p.T, H4 = 4 * H;
  float* ws = sm;                                  // [H][K + 4]: W_hh of this CTA's gate rows, k = gate * UT + unit
  float* ds = ws + (long long)H * pitch;           // [kMB][K + 4]: dgates_t of this CTA's units
  float* part = ds + kMB * pitch;                  // [PARTS][CELLS]
  float* dcs = part + kThreads;                    // [sub][CELLS]: dc carried from step to step
  const int u0 = blockIdx.x * UT, ug = p.ug;
  const int bg0 = blockIdx.y * p.sub * kMB;
  if (threadIdx.x == 0) abort_flag = 0;
  for (int i = threadIdx.x; i < K * H; i += kThreads) {
    const int k = i / H, n = i - k * H, g = k / UT, uu = u0 + (k - g * UT);
    ws[n * pitch + k] = uu < H ? p.w[((long long)g * H + uu) * H + n] : 0.f;
  }
  const int cell_i = threadIdx.x % CELLS, pt = threadIdx.x / CELLS;
  const int cell_m = cell_i / UT, cell_u = cell_i % UT, u = u0 + cell_u;
  for (int s = 0; s < p.sub; s++) {
    const int b = bg0 + s * kMB + cell_m;
    if (pt == 0) dcs[s * CELLS + cell_i] = (u < H && b < p.B && p.dcn != nullptr) ? p.dcn[(long long)b * H + u] : 0.f;
  }
  __syncthreads();
  const int ng_all = H / 4;
  const int lane = threadIdx.x & 31;
  const int per = (ug + PARTS - 1) / PARTS, src0 = pt * per, src1 = min(ug, src0 + per);
  const long long slot_words = (long long)gridDim.y * p.sub * ug * ug * CELLS;
  for (int t = T - 1; t >= 0; t--) {
    for (int s = 0; s < p.sub; s++) {
      const int b0 = bg0 + s * kMB, b = b0 + cell_m;
      const bool live = u < H && b < p.B, mine = live && pt == 0;
      const long long row = (long long)b * T + t;
      unsigned long long* words = p.xch + ((long long)blockIdx.y * p.sub + s) * ug * ug * CELLS;
      float dh = 0.f, ig = 0.f, fg = 0.f, gg = 0.f, og = 0.f, ct = 0.f, cp = 0.f;
      if (mine) {                                  // in flight while the words arrive
        const float* a = p.act + row * H4 + u;
        ig = __ldg(a); fg = __ldg(a + H); gg = __ldg(a + 2 * H); og = __ldg(a + 3 * H);
        ct = __ldg(p.cseq + row * H + u);
        cp = t > 0 ? __ldg(p.cseq + (row - 1) * H + u) : (p.c0 != nullptr ? p.c0[(long long)b * H + u] : 0.f);
        if (p.dout != nullptr) dh = __ldg(p.dout + row * H + u);
      }
      if (t < T - 1) {
        const unsigned long long* in = words + ((t + 1) & 1) * slot_words + (long long)blockIdx.x * ug * CELLS + cell_i;
        const unsigned step = (unsigned)(T - 1 - t);
        float v = 0.f;
        for (int s0 = src0; s0 < src1; s0 += U) {
          unsigned long long w[U];
          unsigned todo = live ? (src1 - s0 >= U ? (1u << U) - 1 : (1u << (src1 - s0)) - 1) : 0u;
          const unsigned all = todo;
          uint64_t t0 = 0;
          for (uint32_t spins = 0; todo != 0; spins++) {
#pragma unroll
            for (int i = 0; i < U; i++)
              if (todo >> i & 1u)
                asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w[i]) : "l"(in + (long long)(s0 + i) * CELLS) : "memory");
#pragma unroll
            for (int i = 0; i < U; i++)
              if ((unsigned)(w[i] >> 32) == step) todo &= ~(1u << i);
            if (todo != 0 && (spins & 0xFF) == 0xFF) {
              if (t0 == 0) t0 = globaltimer_ns();
              if (*(volatile int*)&abort_flag) break;
              if (globaltimer_ns() - t0 > kWaitBudgetNs) {
                *(volatile int*)&abort_flag = 1;
                set_status(p.status, ST_RNN_TIMEOUT, (int)step);
                break;
              }
            }
          }
#pragma unroll
          for (int i = 0; i < U; i++)
            if (all >> i & 1u) v += __uint_as_float((unsigned)w[i]);
        }
        part[threadIdx.x] = v;
        __syncthreads();
        if (*(volatile int*)&abort_flag != 0) return;
        if (mine) {
          v = 0.f;
#pragma unroll
          for (int i = 0; i < PARTS; i++) v += part[i * CELLS + cell_i];
          dh += v;
        }
      } else if (s > 0) {
        __syncthreads();                           // the product of the sub-tile before has read ds
      }
      if (pt == 0) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        if (mine) {
          const float tc = tanhf(ct);
          float* dcv = dcs + s * CELLS + cell_i;
          const float dc = *dcv + dh * og * (1.f - tc * tc);
          d[0] = dc * gg * ig * (1.f - ig);
          d[1] = dc * cp * fg * (1.f - fg);
          d[2] = dc * ig * (1.f - gg * gg);
          d[3] = dh * tc * og * (1.f - og);
          *dcv = dc * fg;
          if (t == 0 && p.dc0 != nullptr) p.dc0[(long long)b * H + u] = dc * fg;
        }
#pragma unroll
        for (int g = 0; g < 4; g++) ds[cell_m * pitch + g * UT + cell_u] = d[g];
        if (mine) {
          float* o = p.dgates + row * H4 + u;
#pragma unroll
          for (int g = 0; g < 4; g++) o[g * H] = d[g];
        }
      }
      __syncthreads();
      if (t == 0) continue;
      unsigned long long* out = words + (t & 1) * slot_words + (long long)blockIdx.x * CELLS;
      const unsigned long long tag = (unsigned long long)(unsigned)(T - t) << 32;
      // a lane takes 4 x 4 sums over all k (lanes that split the contraction cost more in shuffles than they saved, at any H):
      // rows 4 mg .., columns ng + j H / 4, a warp 16 neighbouring columns of all eight rows
      const int mg = lane >> 4;
      for (int ng = (threadIdx.x >> 5) * 16 + (lane & 15); ng < ng_all; ng += kWarps * 16) {
        const float* ap = ds + mg * 4 * pitch;
        const float* wp = ws + ng * pitch;
        unsigned long long acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
#pragma unroll 4
        for (int k = 0; k < K; k += 4) {
          ulonglong2 av[4], wv[4];
#pragma unroll
          for (int i = 0; i < 4; i++) av[i] = *reinterpret_cast<const ulonglong2*>(ap + i * pitch + k);
#pragma unroll
          for (int j = 0; j < 4; j++) wv[j] = *reinterpret_cast<const ulonglong2*>(wp + j * ng_all * pitch + k);
#pragma unroll
          for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
              ffma2(acc[i][j], av[i].x, wv[j].x);
              ffma2(acc[i][j], av[i].y, wv[j].y);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int n = j * ng_all + ng, dest = n / UT;
          unsigned long long* o = out + (long long)dest * ug * CELLS + (n - dest * UT);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float v = __uint_as_float((unsigned)(acc[i][j] & 0xffffffffull)) + __uint_as_float((unsigned)(acc[i][j] >> 32));
            const int m = mg * 4 + i;
            if (b0 + m < p.B)
              asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(o + m * UT), "l"((unsigned long long)__float_as_uint(v) | tag) : "memory");
          }
        }
      }
    }
  }
}

constexpr int kSms = 148;       // of a whole B200; also the words of the flags' scratch
// SMs of the current device: all CTAs of a cooperative launch need one each.  (No device, as in host-side tests: a whole B200.)
int device_sms() {
  int dev, n;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return kSms;
  }
  return n < kSms ? n : kSms;
}
constexpr long long kMaxSmem = 227 * 1024 - 16;      // what a block may take, less the kernels' static abort flag
// Each sub-tile costs a group of CTAs about 1.9 us forward and 2.9 us backward (H = 512); beyond 32 of them the
// step-by-step GEMMs fill the GPU themselves (forward + backward over 8 steps at H = 512: B = 1024, 32
// sub-tiles, 3.4 ms against 4.6 ms step by step; B = 2048, 7.4 against 6.1).
constexpr int kMaxSub = 32;
constexpr long long kScatterBytes = 128ll << 20;

long long fwd_smem(int ut, int H, int parts) {
  return 4ll * ((4ll * ut + kMB) * (H + 4) + (long long)parts * kWarps * kMB * 4 * ut);
}
int fwd_parts(int ut, int H) { return ut == 16 && fwd_smem(ut, H, 2) > kMaxSmem ? 1 : 2; }
long long bwd_smem(int ut, int H, int sub) {
  return 4ll * (((long long)ut + kMB) * (4ll * H + 4) + (long long)kWarps * kMB * ut + (long long)sub * kMB * ut);
}

long long bwd_scatter_smem(int ut, int H, int sub) {
  return 4ll * (((long long)H + kMB) * (4ll * ut + 4) + kThreads + (long long)sub * kMB * ut);
}
// Words of the exchange of the scattered backward, 0 where the gathered one runs: the scattered one is the faster at every size,
// but its words (H = 512: 256 KB a sequence) would be a large part of the memory, and of L2, at thousands of sequences.
long long bwd_words(int ut, int ug, int groups, int sub, int H) {
  const long long words = 2ll * groups * sub * ug * ug * kMB * ut;
  return 8 * words <= kScatterBytes && bwd_scatter_smem(ut, H, sub) <= kMaxSmem ? words : 0;
}

// Units per CTA, unit slices, groups of sequences and sub-tiles per group; false when the layer does
// not fit (the weight slices of `sms` CTAs, or the exchange tile, exceed shared memory).
// Large UT keeps the exchanged tile small against the resident weight; it is halved while that
// gives more CTAs than half of the SMs would otherwise see.
bool plan(int sms, int B, int H, bool bwd, int* ut, int* ug, int* groups, int* sub) {
  if (H % 4 != 0 || H < 4) return false;
  const int tiles = (B + kMB - 1) / kMB;
  int best = 0;
  for (int u = 16; u >= 4; u >>= 1) {
    const int slices = (H + u - 1) / u;
    if (slices > sms) break;                      // smaller u only makes more slices
    const int g = tiles < sms / slices ? tiles : sms / slices;
    const int s = (tiles + g - 1) / g;
    const long long need = bwd ? bwd_smem(u, H, s) : fwd_smem(u, H, fwd_parts(u, H));
    if (need > kMaxSmem || s > kMaxSub) continue;
    *ut = u; *ug = slices; *sub = s; *groups = (tiles + s - 1) / s;
    best = u;
    if ((long long)slices * *groups >= sms / 2) break;
  }
  return best != 0;
}

template <typename K>
int launch(K kern, const SeqArgs& a, int groups, long long smem, long long words, cudaStream_t s) {
  GB_CUDA_OK(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (words > 0) GB_CUDA_OK(cudaMemsetAsync(a.xch, 0, 8ll * words, s));
  else GB_CUDA_OK(cudaMemsetAsync(a.flags, 0, sizeof(unsigned int) * a.ug * groups, s));
  void* args[] = {(void*)&a};
  GB_CUDA_OK(cudaLaunchCooperativeKernel((const void*)kern, dim3(a.ug, groups), dim3(kThreads), args, (size_t)smem, s));
  return gbh::E_OK;
}

}  // namespace

// Dynamic shared memory of a CTA of either direction, 0 when the layer does not fit (for tests).
GB_EXPORT int gb_lstm_seq_smem(int B, int H, int bwd) {
  int ut, ug, groups, sub;
  if (B <= 0 || !plan(kSms, B, H, bwd != 0, &ut, &ug, &groups, &sub)) return 0;
  return (int)(bwd ? bwd_smem(ut, H, sub) : fwd_smem(ut, H, fwd_parts(ut, H)));
}
// 1 when both directions of an LSTM layer of this size run as persistent kernels on that many SMs ...
GB_EXPORT int gb_lstm_seq_fits_on(int sms, int B, int H) {
  int ut, ug, groups, sub;
  return B > 0 && plan(sms, B, H, false, &ut, &ug, &groups, &sub) && plan(sms, B, H, true, &ut, &ug, &groups, &sub) ? 1 : 0;
}
// ... and on the current device.
GB_EXPORT int gb_lstm_seq_fits(int B, int H) { return gb_lstm_seq_fits_on(device_sms(), B, H); }

// fp32.  xg (B,T,4H) = x W_ih^T, bias (4H) or null, w = W_hh (4H,H), h0 / c0 (B,H) or null; writes out (B,T,H), whose sequences are
// out_sb elements apart.  For a backward (hprev not null): h_{t-1} of every step in hprev (B,T,H) (a buffer of its own, so that the
// caller of the layer may change out), all cell states in c (B,T,H), and the activated gates in the place of xg.  Without one
// (hprev null): only the last cell state, in c (B,H), which may be c0.  xch: scratch of 2 * B * H 64-bit words, 16-byte aligned.
GB_EXPORT int gb_lstm_seq_fwd(void* xg, const void* bias, const void* w, const void* h0, const void* c0, void* out, long long out_sb,
                              void* hprev, void* c, void* xch, int B, int T, int H, void* stream) {
  if (B <= 0 || T <= 0) return gbh::E_OK;
  SeqArgs a = {};
  int ut, groups;
  if (!plan(device_sms(), B, H, false, &ut, &a.ug, &groups, &a.sub)) {
    gbh::set_error("gb_lstm_seq_fwd: a layer of %d units does not fit", H);
    return gbh::E_TOO_LARGE;
  }
  a.B = B; a.T = T; a.H = H;
  a.w = (const float*)w; a.h0 = (const float*)h0; a.c0 = (const float*)c0;
  a.xch = (unsigned long long*)xch; a.status = gbh::status_ptr();
  a.xg = (float*)xg; a.bias = (const float*)bias;
  a.out = (float*)out; a.out_sb = out_sb; a.hprev = (float*)hprev; a.cseq = (float*)c;
  if (hprev != nullptr && out_sb != (long long)T * H) {
    gbh::set_error("gb_lstm_seq_fwd: a contiguous output is needed where a backward follows");
    return gbh::E_BAD_ARG;
  }
  const int parts = fwd_parts(ut, H);
  const long long smem = fwd_smem(ut, H, parts), words = 2ll * B * H;
  cudaStream_t s = (cudaStream_t)stream;
  if (hprev != nullptr) {
    if (ut == 16 && parts == 1) return launch(lstm_seq_fwd_kernel<16, true, 1>, a, groups, smem, words, s);
    if (ut == 16) return launch(lstm_seq_fwd_kernel<16, true, 2>, a, groups, smem, words, s);
    if (ut == 8) return launch(lstm_seq_fwd_kernel<8, true, 2>, a, groups, smem, words, s);
    return launch(lstm_seq_fwd_kernel<4, true, 2>, a, groups, smem, words, s);
  }
  if (ut == 16 && parts == 1) return launch(lstm_seq_fwd_kernel<16, false, 1>, a, groups, smem, words, s);
  if (ut == 16) return launch(lstm_seq_fwd_kernel<16, false, 2>, a, groups, smem, words, s);
  if (ut == 8) return launch(lstm_seq_fwd_kernel<8, false, 2>, a, groups, smem, words, s);
  return launch(lstm_seq_fwd_kernel<4, false, 2>, a, groups, smem, words, s);
}

// 64-bit words of scratch with which gb_lstm_seq_bwd runs at its fastest (it runs with kSms / 2, too).
GB_EXPORT long long gb_lstm_seq_bwd_words(int B, int H) {
  int ut, ug, groups, sub;
  if (B <= 0 || !plan(device_sms(), B, H, true, &ut, &ug, &groups, &sub)) return 0;
  const long long words = bwd_words(ut, ug, groups, sub, H);
  return words > kSms / 2 ? words : kSms / 2;
}

// Backward of the above (scratch: gb_lstm_seq_bwd_words(B, H) 64-bit words, or kSms / 2 where memory is short: then dgates are
// gathered): dout (B,T,H) or null, dcn (B,H) or null; writes dgates (B,T,4H), the gradient
// of the gate pre-activations, and dc0 (B,H) when not null.
GB_EXPORT int gb_lstm_seq_bwd(const void* w, const void* c0, const void* cseq, const void* act, const void* dout,
                              const void* dcn, void* dgates, void* dc0, void* scratch, long long scratch_words, int B, int T,
                              int H, void* stream) {
  if (B <= 0 || T <= 0) return gbh::E_OK;
  SeqArgs a = {};
  int ut, groups;
  if (!plan(device_sms(), B, H, true, &ut, &a.ug, &groups, &a.sub)) {
    gbh::set_error("gb_lstm_seq_bwd: a layer of %d units does not fit", H);
    return gbh::E_TOO_LARGE;
  }
  a.B = B; a.T = T; a.H = H;
  a.w = (const float*)w; a.c0 = (const float*)c0; a.cseq = (float*)cseq; a.act = (const float*)act;
  a.dout = (const float*)dout; a.dcn = (const float*)dcn; a.dgates = (float*)dgates; a.dc0 = (float*)dc0;
  a.status = gbh::status_ptr();
  cudaStream_t s = (cudaStream_t)stream;
  // A single step exchanges nothing, and of two the words' clear costs more than one exchange gains.  us, scattered | gathered: two steps
  // B = H = 512 132 | 118, 256 x 512 76 | 68, 32 x 512 27.0 | 24.1, 64 x 64 11.5 | 9.8, 256 x 256 26.6 | 28.6; three 203 | 213, 105 | 117,
  // 31.1 | 30.9, 11.5 | 12.6, 34.8 | 43.2.
  const long long words = T > 2 ? bwd_words(ut, a.ug, groups, a.sub, H) : 0;
  if (scratch_words < kSms / 2) {
    gbh::set_error("gb_lstm_seq_bwd: %d words of scratch are needed", kSms / 2);
    return gbh::E_BAD_ARG;
  }
  if (words > 0 && scratch_words >= words) {
    a.xch = (unsigned long long*)scratch;
    const long long smem = bwd_scatter_smem(ut, H, a.sub);
    const int parts = kThreads / (kMB * ut);
    const bool deep = (a.ug + parts - 1) / parts > 8;
    if (ut == 16) return deep ? launch(lstm_seq_bwd_scatter_kernel<16, 16>, a, groups, smem, words, s) : launch(lstm_seq_bwd_scatter_kernel<16, 8>, a, groups, smem, words, s);
    if (ut == 8) return deep ? launch(lstm_seq_bwd_scatter_kernel<8, 16>, a, groups, smem, words, s) : launch(lstm_seq_bwd_scatter_kernel<8, 8>, a, groups, smem, words, s);
    return deep ? launch(lstm_seq_bwd_scatter_kernel<4, 16>, a, groups, smem, words, s) : launch(lstm_seq_bwd_scatter_kernel<4, 8>, a, groups, smem, words, s);
  }
  a.flags = (unsigned int*)scratch;
  const long long smem = bwd_smem(ut, H, a.sub);
  if (ut == 16) return launch(lstm_seq_bwd_kernel<16>, a, groups, smem, 0, s);
  if (ut == 8) return launch(lstm_seq_bwd_kernel<8>, a, groups, smem, 0, s);
  return launch(lstm_seq_bwd_kernel<4>, a, groups, smem, 0, s);
}
