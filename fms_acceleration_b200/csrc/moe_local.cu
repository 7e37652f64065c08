// The launches of a mixture-of-experts layer on one GPU in one call per direction (no low-rank factors, no token slices): plan,
// dispatch, grouped GEMMs, activation, combine.  From Python the seventeen launches of a training pass cost the host some
// 25 us each, more than their kernels take for a few hundred tokens.  250 tokens, 40 experts of 1536 x 512, top 8, forward and
// backward: 472 -> 288 us a pass.
#include "common.cuh"

extern "C" {
int fmsb_moe_plan(const int*, long long, int, int, int, int, int*, void* const*, void* const*, unsigned, int*, int*, int*, int*,
                  int*, int*, int*, int*, cudaStream_t);
int fmsb_moe_zero_pad(void*, long long, int, const int*, const int*, int, int, cudaStream_t);
int fmsb_moe_dispatch(const void*, long long, const int*, const int*, const float*, long long, int, int, int, void* const*,
                      long long, int, int, cudaStream_t);
int fmsb_moe_dispatch_dot(const void*, long long, const int*, const float*, long long, int, int, const void*, long long, void*,
                          long long, float*, int, cudaStream_t);
int fmsb_moe_combine(void* const*, long long, const int*, const int*, const float*, long long, int, int, int, void*, long long,
                     int, int, cudaStream_t);
int fmsb_glu_fwd(const void*, const void*, void*, int, int, long long, long long, long long, int, int, const int*, cudaStream_t);
int fmsb_glu_bwd(const void*, const void*, const void*, void*, void*, void*, int, int, long long, long long, long long, long long,
                 long long, long long, int, int, const int*, cudaStream_t);
int fmsb_grouped_gemm2(const void*, long long, const void*, long long, int, int, const void*, int, const void*, long long,
                       const void*, long long, int, void*, long long, int, const void*, long long, int, float, float, int, int,
                       int, int, int, int, const int*, long long, long long, long long, int, int*, cudaStream_t);
}

namespace {
// tile width of a grouped product with n output columns (with n_split: a divisor of one of the two side-by-side halves)
int tile_n(int n, int n_split) {
  const int m = n_split ? n_split : n;
  int bn = m >= 192 ? 256 : (m > 64 ? 128 : 64);
  if (n_split && n_split % bn) bn = n_split % 128 == 0 ? 128 : 64;
  return bn;
}

struct Group {  // what the grouped products of one call share
  const int* seg_off;
  int E;
  long long cap;
  int fmt, max_ctas;
  int* status;
  cudaStream_t stream;

  // D [cap, n] = A [cap, K] . B_g (+ A2 . B2_g); B stored [E * K, n] (b_mn) or [E * n, K]; B_alt: the right half of D, rows
  // as far apart as B's
  int rows(const void* A, long long lda, const void* B, long long ldb, int K, int b_mn, const void* B_alt, int n_split,
           const void* A2, long long lda2, const void* B2, long long ldb2, int K2, void* D, long long ldd, int n) const {
    return fmsb_grouped_gemm2(A, lda, B, ldb, K, b_mn, B_alt, n_split, A2, lda2, B2, ldb2, K2, D, ldd, 0, nullptr, 0, 0,
                              1.f, 0.f, 0, n, fmt, tile_n(n, n_split), 1, E, seg_off, 0, cap, (long long)E * (b_mn ? K : n),
                              max_ctas, status, stream);
  }
  // D [E, m, n] = A_g^T . B_g over the rows of every segment
  int weights(const void* A, long long lda, const void* B, long long ldb, void* D, int m, int n) const {
    return fmsb_grouped_gemm2(A, lda, B, ldb, 64, 1, nullptr, 0, nullptr, 0, nullptr, 0, 0, D, n, 0, nullptr, 0, 0, 1.f, 0.f, m,
                              n, fmt, tile_n(n, 0), 2, E, seg_off, (long long)m * n, cap, cap, max_ctas, status, stream);
  }
};
}  // namespace

#define FMSB_TRY(call) do { if (int rc_ = (call)) return rc_; } while (0)

// x [T, H]; idx, gates [T, k]; w1, w3 [E, H, I] with rows ld13 apart, w2 [E, I, H] with rows ld2 apart.
// ws: 3 E + max(1, ceil(T k / 1024)) E ints.  seg_off [E + 1], seg_cnt [E], dest_row [T, k]; Xs, Ys [cap, H], gu [cap, 2 I], hs [cap, I]; out [T, H].
extern "C" int fmsb_moe_local_fwd(const void* x, long long ldx, const int* idx, const float* gates, long long T, int k, int H,
                                  int I, int E, const void* w1, const void* w3, long long ld13, const void* w2, long long ld2,
                                  int act, int* ws, int* seg_off, int* seg_cnt, int* dest_row, int cap, void* Xs, void* gu,
                                  void* hs, void* Ys, void* out, int* needed, int* overflow, int fmt, int max_ctas, int* status, cudaStream_t stream) {
  FMSB_TRY((int)cudaMemsetAsync(ws, 0, sizeof(int) * E, stream));
  FMSB_TRY(fmsb_moe_plan(idx, T * k, E, 0, 1, cap, ws, nullptr, nullptr, 0, seg_off, seg_cnt, ws + E, dest_row, needed,
                         ws + 3 * E, overflow, status, stream));
  FMSB_TRY(fmsb_moe_zero_pad(Xs, H, H, seg_off, seg_cnt, E, fmt, stream));
  void* xs[1] = {Xs};
  FMSB_TRY(fmsb_moe_dispatch(x, ldx, idx, dest_row, nullptr, T * k, k, H, E, xs, H, 1, fmt, stream));
  const Group g{seg_off, E, cap, fmt, max_ctas, status, stream};
  uint16_t* gu16 = (uint16_t*)gu;
  FMSB_TRY(g.rows(Xs, H, w1, ld13, H, 1, w3, I, nullptr, 0, nullptr, 0, 0, gu, 2LL * I, 2 * I));
  FMSB_TRY(fmsb_glu_fwd(gu16, gu16 + I, hs, cap, I, 2LL * I, 2LL * I, I, act, fmt, seg_off + E, stream));
  FMSB_TRY(g.rows(hs, I, w2, ld2, I, 1, nullptr, 0, nullptr, 0, nullptr, 0, 0, Ys, H, H));
  void* ys[1] = {Ys};
  return fmsb_moe_combine(ys, H, idx, dest_row, gates, T, k, H, E, out, H, 1, fmt, stream);
}

// dout [T, H].  gu is overwritten with the pre-activation gradients.  hs, dhs [cap, I], dYs, dXs [cap, H] scratch; dw1, dw3
// [E, H, I], dw2 [E, I, H] (all or none null); dgate [T, k]; dx [T, H].
extern "C" int fmsb_moe_local_bwd(const void* dout, long long ldd, const int* idx, const float* gates, const int* seg_off,
                                  const int* seg_cnt, const int* dest_row, const void* Xs, void* gu, const void* Ys, long long T,
                                  int k, int H, int I, int E, const void* w1, const void* w3, long long ld13, const void* w2,
                                  long long ld2, int act, int cap, void* dYs, void* hs, void* dhs, void* dXs, float* dgate,
                                  void* dx, void* dw1, void* dw3, void* dw2, int fmt, int max_ctas, int* status, cudaStream_t stream) {
  FMSB_TRY(fmsb_moe_zero_pad(dYs, H, H, seg_off, seg_cnt, E, fmt, stream));
  FMSB_TRY(fmsb_moe_dispatch_dot(dout, ldd, dest_row, gates, T, k, H, Ys, H, dYs, H, dgate, fmt, stream));
  const Group g{seg_off, E, cap, fmt, max_ctas, status, stream};
  uint16_t* gu16 = (uint16_t*)gu;
  if (dw2 != nullptr) {
    FMSB_TRY(fmsb_glu_fwd(gu16, gu16 + I, hs, cap, I, 2LL * I, 2LL * I, I, act, fmt, seg_off + E, stream));
    FMSB_TRY(g.weights(hs, I, dYs, H, dw2, I, H));
  }
  FMSB_TRY(g.rows(dYs, H, w2, ld2, H, 0, nullptr, 0, nullptr, 0, nullptr, 0, 0, dhs, I, I));
  FMSB_TRY(fmsb_glu_bwd(dhs, gu16, gu16 + I, gu16, gu16 + I, nullptr, cap, I, I, 2LL * I, 2LL * I, 2LL * I, 2LL * I, 0, act, fmt,
                        seg_off + E, stream));
  if (dw2 != nullptr) {
    FMSB_TRY(g.weights(Xs, H, gu16, 2LL * I, dw1, H, I));
    FMSB_TRY(g.weights(Xs, H, gu16 + I, 2LL * I, dw3, H, I));
  }
  FMSB_TRY(g.rows(gu16, 2LL * I, w1, ld13, I, 0, nullptr, 0, gu16 + I, 2LL * I, w3, ld13, I, dXs, H, H));
  void* xs[1] = {dXs};
  return fmsb_moe_combine(xs, H, idx, dest_row, nullptr, T, k, H, E, dx, H, 1, fmt, stream);
}
