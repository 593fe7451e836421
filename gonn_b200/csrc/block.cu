// One transformer block without a tape: the launches of its seven kernels from one native call.
//
// A block evaluated operator by operator costs seven Python operators (tape node, argument conversion, one
// ctypes call each): 290 us of host time for kernels that take 58 us at 77 tokens of the 768-wide model.  The
// kernels and their order are those of the operators: norm, QKV product, attention, output product + residual,
// norm, first product + activation, second product + residual.  The pre-activation, which only a backward would
// read, is not stored (134 MB a layer at 8192 tokens x 8192).
#include "common.cuh"

extern "C" {
int gb_gemm16(const void* A, const void* B, void* C, const void* bias, int bias_f32, void* aux, int M, int N, int K, int batch,
              int transA, int transB, long long lda, long long ldb, long long ldc, long long ldaux, long long sA, long long sB,
              long long sC, long long sAux, int in_dtype, int out_dtype, int act, int aux_mode, int beta, float alpha, int force_bn,
              void* workspace, long long workspace_bytes, void* stream);
int gb_norm_fwd(int kind, int dtype, int wdtype, const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                long long rows, int D, float eps, void* stream);
int gb_flash_fwd(int dtype, const void* q, const void* k, const void* v, void* o, float* lse, int B, int H, int Sq, int Sk, int D,
                 long long q_sb, long long q_ss, long long q_sh, long long k_sb, long long k_ss, long long k_sh, long long v_sb,
                 long long v_ss, long long v_sh, long long o_sb, long long o_ss, long long o_sh, float scale, int causal, void* stream);
}

namespace {

// the caller's array of words, in this order (nn/block.py)
struct BlockArgs {
  long long dtype;         // 0 bf16, 1 fp16
  long long B, S, E, H, F;
  long long rms, pre_norm, causal, act;
  long long x, y;          // (B, S, E)
  long long n1w, n1b, n2w, n2b;
  long long wqkv, bqkv, wo, bo, w1, b1, w2, b2;   // biases may be null
  long long ws, ws_bytes;
};
constexpr int kWords = sizeof(BlockArgs) / 8;

long long align16(long long n) { return (n + 15) / 16 * 16; }
long long act_bytes(long long B, long long S, long long E) { return align16(2 * B * S * E); }

}  // namespace

// Bytes of scratch of gb_block_fwd (16-byte aligned).
GB_EXPORT long long gb_block_ws(int B, int S, int E, int H, int F) {
  const long long rows = (long long)B * S, wide = 3LL * E > F ? 3LL * E : F;
  return 2 * act_bytes(B, S, E) + align16(2 * rows * wide) + align16(4LL * B * H * S) + 2 * align16(4 * rows);
}

GB_EXPORT int gb_block_fwd(const long long* words, int n, float eps1, float eps2, float scale, void* stream) {
  if (n != kWords) {
    gbh::set_error("gb_block_fwd: %d argument words, expected %d", n, kWords);
    return gbh::E_BAD_ARG;
  }
  BlockArgs a;
  memcpy(&a, words, sizeof(a));
  if (a.ws_bytes < gb_block_ws((int)a.B, (int)a.S, (int)a.E, (int)a.H, (int)a.F)) {
    gbh::set_error("gb_block_fwd: workspace too small");
    return gbh::E_BAD_ARG;
  }
  const int dt = (int)a.dtype, E = (int)a.E, F = (int)a.F, D = E / (int)a.H, rows = (int)(a.B * a.S);
  auto P = [](long long p) { return (void*)p; };
  char* w = (char*)P(a.ws);
  char* buf_n = w;  w += act_bytes(a.B, a.S, E);                     // norm output, attention output
  char* buf_x = w;  w += act_bytes(a.B, a.S, E);                     // the residual stream between the halves
  char* buf_w = w;  w += align16(2LL * rows * (3 * E > F ? 3 * E : F));   // QKV, hidden activations
  float* lse = (float*)w;  w += align16(4LL * a.B * a.H * a.S);
  float* mean = (float*)w;  w += align16(4LL * rows);
  float* rstd = (float*)w;
  int rc;
  auto norm = [&](const void* x, long long g, long long b, void* y, float eps) {
    return gb_norm_fwd((int)a.rms, dt, dt, x, P(g), P(b), y, a.rms ? nullptr : mean, rstd, rows, E, eps, stream);
  };
  // y = act(x W^T + b) (+ res); aux mode 1: residual
  auto linear = [&](const void* x, long long W, long long b, void* y, int N, int K, int act, const void* res) {
    return gb_gemm16(x, P(W), y, P(b), 0, const_cast<void*>(res), rows, N, K, 1, 0, 1, K, K, N, N, 0, 0, 0, 0, dt, dt, act,
                     res ? 1 : 0, 0, 1.f, 0, nullptr, 0, stream);
  };
  const void* x = P(a.x);
  const void* in = x;
  if (a.pre_norm) {
    if ((rc = norm(x, a.n1w, a.n1b, buf_n, eps1))) return rc;
    in = buf_n;
  }
  if ((rc = linear(in, a.wqkv, a.bqkv, buf_w, 3 * E, E, 0, nullptr))) return rc;
  const long long sb = 3LL * E * a.S, ss = 3LL * E;
  if ((rc = gb_flash_fwd(dt, buf_w, buf_w + 2LL * E, buf_w + 4LL * E, buf_n, lse, (int)a.B, (int)a.H, (int)a.S, (int)a.S, D, sb, ss, D,
                         sb, ss, D, sb, ss, D, (long long)E * a.S, E, D, scale, (int)a.causal, stream)))
    return rc;
  if ((rc = linear(buf_n, a.wo, a.bo, buf_x, E, E, 0, x))) return rc;
  if (a.pre_norm) {
    if ((rc = norm(buf_x, a.n2w, a.n2b, buf_n, eps2))) return rc;
    if ((rc = linear(buf_n, a.w1, a.b1, buf_w, F, E, (int)a.act, nullptr))) return rc;
    return linear(buf_w, a.w2, a.b2, P(a.y), E, F, 0, buf_x);
  }
  if ((rc = norm(buf_x, a.n1w, a.n1b, buf_n, eps1))) return rc;
  if ((rc = linear(buf_n, a.w1, a.b1, buf_w, F, E, (int)a.act, nullptr))) return rc;
  if ((rc = linear(buf_w, a.w2, a.b2, buf_x, E, F, 0, buf_n))) return rc;
  return norm(buf_x, a.n2w, a.n2b, P(a.y), eps2);
}

// Blocks one after another, as gb_block_fwd takes them: argument words and (eps1, eps2, scale) of counts[0] of them in `words` and
// `scalars`, which have room for `room`.  While counts[2] says that there are more, `more` is called once these are launched and leaves
// the next ones there (none of them by not coming so far).  So the first kernel starts when the first block is known, and the GPU
// works while the caller looks at the others.  counts[1]: how many are launched.
GB_EXPORT int gb_stack_fwd(void (*more)(), int* counts, const long long* words, const float* scalars, int n, int room, void* stream) {
  for (counts[1] = 0; counts[0] > 0 && counts[0] <= room;) {
    for (int i = 0; i < counts[0]; i++, counts[1]++) {
      const int rc = gb_block_fwd(words + (long long)i * n, n, scalars[3 * i], scalars[3 * i + 1], scalars[3 * i + 2], stream);
      if (rc) return rc;
    }
    if (counts[2] == 0) break;
    counts[0] = counts[2] = 0;
    more();
  }
  return gbh::E_OK;
}
