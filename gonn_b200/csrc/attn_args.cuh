// Arguments of the general attention kernels and the dropout draw they share (attn_general.cu, attn_f64.cu).
#pragma once
#include "common.cuh"

namespace gba {

enum { MODE_FWD = 0, MODE_DQ = 1, MODE_DKV = 2 };

struct GArgs {
  const void *Q, *K, *V, *dO;
  void *O, *dQ, *dK, *dV;
  void* LSE;             // [B, H, Tq], natural log; in the compute type (fp32, or fp64 for fp64 tensors)
  void* Delta;           // [B, H, Tq], same type
  long long q_s[3], k_s[3], v_s[3], o_s[3], g_s[3], dq_s[3], dk_s[3], dv_s[3];  // (b, s, h) element strides
  int B, H, Tq, Tk, D;
  double scale;
  int causal;
  const float* mask;            // [Tq, Tk] additive, or null
  const unsigned char* kpm;     // [B, Tk], 1 = padded key, or null
  double p_drop;
  unsigned long long seed;
  // fp64, head size <= 64, optional: dS^T (B * H, Tk, Tq) with both lengths rounded up to 64, written by the dK / dV
  // role; the dQ role is then its product with K
  double* dS;
  long long ds_rows, ds_ld;
};

__device__ __forceinline__ uint4 philox(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; r++) {
    uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += W0;
    key.y += W1;
  }
  return ctr;
}
// One Philox call serves the four queries 4g .. 4g+3 against key k: counter (g, k, bh), query q takes
// word q % 4.  A warp's four query rows (forward, dQ) start at a multiple of four, so there one call
// per lane and tile covers all four rows; the dK/dV role (rows are keys) draws once per cell.
__device__ __forceinline__ uint4 keep_draw(const GArgs& a, int bh, int qgroup, int k) {
  return philox(make_uint4((uint32_t)qgroup, (uint32_t)k, (uint32_t)bh, 0u),
                make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32)));
}
__device__ __forceinline__ uint32_t draw_word(const uint4& r, int i) {
  return i == 0 ? r.x : i == 1 ? r.y : i == 2 ? r.z : r.w;
}
__device__ __forceinline__ bool keep_cell(const GArgs& a, int bh, int q, int k, uint32_t thresh) {
  return draw_word(keep_draw(a, bh, q >> 2, k), q & 3) >= thresh;
}

// fp64, head size <= 64 (attn_f64.cu); mode 0, 1 or 2.
constexpr int kF64MaxHead = 64;
int launch_f64(int mode, const GArgs& a, cudaStream_t s);

}  // namespace gba
