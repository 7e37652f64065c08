// Chunked state-space-duality scan with its decay matrices kept on the chip (chunk 256, head dimension 64, state 128;
// other shapes take the batched products of gemm_tcgen05.cu and the passes of mamba_scan.cu).
//
// Per chunk c and head h, with L the within-chunk cumulative sum of dt*A and CB = C B^T (shared by the heads of a group):
//
//   G[t, s]  = CB[t, s] exp(L_t - L_s) dt_s          (s <= t, else 0)
//   y        = G x + exp(L_t) (C Hprev^T) + D x       Hprev: state entering the chunk
//   S        = (x w)^T B,   w = exp(L_last - L) dt     what the chunk adds to the state
//   dx       = G^T dy + w (B dS^T) + D dy              dS: gradient of the state leaving the chunk
//   dHprev   = (exp(L) dy)^T C,   dC = (exp(L) dy) Hprev + dCB B,   dB = (x w) dS + dCB^T C
//   dCB      = sum over heads of (dy x^T) o exp(L_t - L_s) dt_s
//
// Written as separate products these cost a [chunks, heads, 256, 256] 16-bit matrix (2.7 GB per layer at 65536 tokens)
// through memory several times and fp32 copies of every [T, heads, 64] product.  Here G is built in registers
// from CB (held as 16-bit pairs, 64 registers a thread) and written to tensor memory as the A operand of G x, like the
// probabilities of an attention kernel; scaled copies of x and dy exist only in shared memory; the epilogues add the
// terms and take the row dot products.  What is left is bound by reading x / dy and writing y / dx once.
//
// Roles (320 threads; the scan kernel's differ, see there): warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 compute (lane quarter
// warp % 4, column half (warp - 2) / 4).  Every wait is bounded.
#include <type_traits>

#include "common.cuh"

namespace fmsb {
namespace ssdf {

constexpr int CQ = 256;  // chunk
constexpr int CP = 64;   // head dimension
constexpr int CN = 128;  // state
constexpr int kTile = 128 * 128;      // bytes of a [128 x 64] 16-bit tile
constexpr float kSplitLimit = 60.f;   // |exponent| across eight columns below which the decay factorises safely

struct ScanParams {
  int nc, nh, G, hp;   // hp: heads per CTA
  const float* Lt;     // [nc, nh, 256]
  const float* dtt;    // [nc, nh, 256]
  const float* D;      // [nh]
  float* red;          // MODE 1: [nc, nh, 256]; MODE 2: three of them (dy.x, w x.(B dS^T), x.(G^T dy))
  float* S;            // state kernel: [nc, nh, 64, 128]
  float* part;         // partial sums over head splits
  int wmode;           // state kernel: 0 rows scaled by exp(L_last - L) dt, 1 by exp(L)
  int T;
  int* status;
};

__device__ __forceinline__ void compute_sync(int id) { asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory"); }

template <int FMT>
__device__ __forceinline__ void unpack2(uint32_t w, float& a, float& b) {
  if (FMT == 1) {
    a = __uint_as_float(w << 16);
    b = __uint_as_float(w & 0xffff0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    a = f.x;
    b = f.y;
  }
}
template <int FMT>
__device__ __forceinline__ uint32_t pack2f(float a, float b) {
  return FMT == 1 ? pack_bf16x2(a, b) : pack_f16x2(a, b);
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint32_t swz(int r, int c16) { return static_cast<uint32_t>(r * 128 + ((c16 ^ (r & 7)) << 4)); }

// Per-head scalars of a chunk in shared memory, three sets (a set is rewritten only after every compute warp has passed
// the barrier that follows its last use).  The decay of eight neighbouring positions is factorised around their first
// one: exp(L_t - L_s) dt_s = exp(ref_t - ref_s) exp(L_t - ref_t) (exp(ref_s - L_s) dt_s), one exponential per row and eight
// columns; `ok` (one flag per 32 positions) says whether the exponents are moderate enough for that, otherwise every element
// of the head takes its own exponential.  One branch per head: a test per eight columns kept the loads of the next ones from
// being issued.
// All modes of the scan kernel multiply the same factors in the same order, (CB (e rf_t)) cf_s: the gradient of the decay is
// a difference of sums over rows (mode 1) and over columns (mode 2) of dG o G, which cancels only between two G that are
// equal in every bit.  Mode 2 with factors around its own rows rounded about one element in 10^4 differently, and dA of one
// input in twenty was 1.8 times as far from 64 bits as the general path's (0.0038 against 0.0021).
struct HeadScalars {
  float L[CQ];
  float d[CQ];
  float cf[CQ];        // as column s: exp(ref_s - L_s) dt_s
  float rf[CQ];        // as row t: exp(L_t - ref_t)
  float ref[CQ / 8];   // L of every eighth position
  int ok[8];
  unsigned zero[8];    // MODE 2: one bit per position with dt = 0
};

// MODE 2 takes 1 for a step size of 0.  ddt is the derivative of products with dt by dt, taken as the product over dt: where
// dt is 0 the products without it are that derivative, and everything else leaves such a position out (`zero`).
template <int MODE>
__device__ __forceinline__ void publish(HeadScalars& hs, int i, float L, float d) {
  const int lane = i & 31;
  if (MODE == 2) {
    const unsigned zero = __ballot_sync(0xffffffffu, d == 0.f);
    if (lane == 0) hs.zero[i >> 5] = zero;
    if (d == 0.f) d = 1.f;
  }
  const float ref = __shfl_sync(0xffffffffu, L, lane & ~7), last = __shfl_sync(0xffffffffu, L, lane | 7);
  hs.L[i] = L;
  hs.d[i] = d;
  hs.cf[i] = __expf(ref - L) * d;
  if (MODE <= 2) hs.rf[i] = __expf(L - ref);
  if ((lane & 7) == 0) hs.ref[i >> 3] = L;
  const int ok = __all_sync(0xffffffffu, fabsf(ref - last) < kSplitLimit);
  if (lane == 0) hs.ok[i >> 5] = ok;
}
__device__ __forceinline__ bool all_ok(const HeadScalars& hs) {
  const int4 a = *reinterpret_cast<const int4*>(&hs.ok[0]), b = *reinterpret_cast<const int4*>(&hs.ok[4]);
  return (a.x & a.y & a.z & a.w & b.x & b.y & b.z & b.w) != 0;
}

// ----------------------------------------------------------------------------------------
// Scan kernel.  grid (nc, G * splits): one chunk, hp heads in turn, each head's two 128-row tiles as two units.
//   MODE 0: rows t; R = C, columns B; V = x, H = Hprev; out = y
//   MODE 1: the same products, out = dy . (G x + exp(L) C Hprev^T) per row (E = dy)
//   MODE 2: rows s; R = B, columns C; V = dy, H = dS; out = dx and three row dot products (E = x)
// Both tiles in one CTA read V and H once (one tile per CTA read them 1.5 and 2 times) and are each other's second
// buffer: while the tensor core works on unit w, the compute warps build G of unit w + 1, then drain unit w.
// Tensor memory: G of the two tiles 64 + 128 columns (16-bit pairs), accumulators 2 x (64 + 64) from column 256.
// 384 threads: warps 0 and 1 as above, 2 and 3 idle, 4-11 compute with 232 registers (C B^T is 96 of them).
// 16384 tokens, 80 heads (one tile per CTA, 168 registers -> this): y 331 -> 146 us, dots 332 -> 142, dx 413 -> 194 us (183
// before it took the factors of the other modes and looked at rows with dt = 0); reading and writing everything once would
// take 63 us at the copy rate.
// ----------------------------------------------------------------------------------------
constexpr int kScanThreads = 384;
constexpr int kScanRegsMain = 40, kScanRegsCompute = 232;  // 128 * 40 + 256 * 232 = 384 * 168
constexpr int kScanStage = 3 * kTile;  // V (256 rows), H (64 x 128)
constexpr int kScanSmem = 4 * kTile + 2 * kScanStage + 3 * kTile + 3 * (int)sizeof(HeadScalars) + 3 * 3 * 128 * 4 + 1024 + 256;

__device__ __forceinline__ void pair_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(quarter + 2) : "memory"); }

template <int MODE, int FMT>
__global__ void __launch_bounds__(kScanThreads, 1)
ssd_scan_kernel(const __grid_constant__ CUtensorMap tmR, const __grid_constant__ CUtensorMap tmCol,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmH,
                const __grid_constant__ CUtensorMap tmE, const __grid_constant__ CUtensorMap tmOut, const ScanParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  auto sR = [&](int t) { return base + t * 2 * kTile; };  // [tile][64-column half]
  auto sV = [&](int s) { return base + 4 * kTile + s * kScanStage; };
  auto sH = [&](int s) { return sV(s) + 2 * kTile; };
  const uint32_t sCol = sV(0);  // prologue only: [tile][half], 64 KB of the 96 KB of the stages
  auto sE = [&](int e) { return base + 4 * kTile + 2 * kScanStage + e * kTile; };  // rows in (E) and out, ring of 3
  const uint32_t scal = sE(3);
  const uint32_t dots = scal + 3 * (uint32_t)sizeof(HeadScalars);
  const uint32_t bars = dots + 3 * 3 * 128 * 4;
  const uint32_t bar_r = bars, bar_cb = bars + 8u;
  auto full = [&](int s) { return bars + 16u + 8u * s; };
  auto empty = [&](int s) { return bars + 32u + 8u * s; };
  auto g_full = [&](int u) { return bars + 48u + 8u * u; };
  auto acc_full = [&](int u) { return bars + 64u + 8u * u; };
  auto e_full = [&](int e) { return bars + 80u + 8u * e; };
  auto e_empty = [&](int e) { return bars + 104u + 8u * e; };
  const uint32_t holder = bars + 128u;
  HeadScalars* hs = reinterpret_cast<HeadScalars*>(smem_raw + (scal - smem_u32(smem_raw)));
  float* sdot = reinterpret_cast<float*>(smem_raw + (dots - smem_u32(smem_raw)));  // [3][3][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x;
  const int hpg = p.nh / p.G, spg = gridDim.y / p.G;
  const int g = blockIdx.y / spg;
  const int h_begin = g * hpg + (blockIdx.y % spg) * p.hp;
  const int n_heads = min(p.hp, (g + 1) * hpg - h_begin);
  // contraction tiles of row tile u: kt0(u) .. kt0(u) + nks(u) - 1; the first 128-column block of C B^T it owns
  auto kt0 = [](int u) { return MODE == 2 ? u : 0; };
  auto nks = [](int u) { return MODE == 2 ? 2 - u : u + 1; };
  auto cb0 = [](int u) { return u == 0 ? 0 : (MODE == 2 ? 2 : 1); };

  if (warp == 1 && lane == 0) {
    mbar_init(bar_r, 1);
    mbar_init(bar_cb, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), MODE == 1 ? 1 : 8);
      mbar_init(g_full(s), 8);
      mbar_init(acc_full(s), 1);
    }
    for (int e = 0; e < 3; ++e) {
      mbar_init(e_full(e), 1);
      mbar_init(e_empty(e), 4);
    }
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(holder));
  auto tG = [&](int u) { return tmem + 64u * cb0(u); };
  auto tAcc = [&](int u) { return tmem + 256u + 128u * u; };  // [G V: 64 | R H^T: 64]

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kScanRegsMain));
    if (warp == 0 && lane == 0) {
      mbar_expect_tx(bar_r, 8 * kTile);
      for (int t = 0; t < 2; ++t)
        for (int k = 0; k < 2; ++k) {
          tma_load_2d(sR(t) + k * kTile, &tmR, bar_r, g * CN + 64 * k, c * CQ + t * 128);
          tma_load_2d(sCol + (2 * t + k) * kTile, &tmCol, bar_r, g * CN + 64 * k, c * CQ + t * 128);
        }
      auto load_e = [&](int w) {  // this CTA's own rows of unit w
        const int e = w % 3;
        if (!mbar_wait(e_empty(e), ((w / 3) & 1) ^ 1u, p.status, kTimeoutProducer)) return false;
        mbar_expect_tx(e_full(e), kTile);
        tma_load_2d(sE(e), &tmE, e_full(e), (h_begin + (w >> 1)) * CP, c * CQ + (w & 1) * 128);
        return true;
      };
      bool ok = true;
      if (MODE != 0) ok = load_e(0) && load_e(1);
      ok = ok && mbar_wait(bar_cb, 0, p.status, kTimeoutProducer);  // the stages are free once C B^T is done
#pragma unroll 1
      for (int it = 0; it < n_heads && ok; ++it) {
        const int s = it & 1, h = h_begin + it;
        if (!mbar_wait(empty(s), ((it >> 1) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(full(s), 3 * kTile);
        for (int i = 0; i < 2; ++i) tma_load_2d(sV(s) + i * kTile, &tmV, full(s), h * CP, c * CQ + i * 128);
        for (int k = 0; k < 2; ++k)
          tma_load_2d(sH(s) + k * (kTile / 2), &tmH, full(s), 64 * k, (c * p.nh + h) * CP);
        if (MODE != 0 && it > 0) ok = load_e(2 * it) && load_e(2 * it + 1);
      }
    } else if (warp == 1 && lane == 0) {
      bool ok = mbar_wait(bar_r, 0, p.status, kTimeoutMma);
      if (ok) {
        tc_fence_after();
        const uint32_t idesc = make_idesc_f16(128, 128, FMT, 0, 0);
#pragma unroll 1
        for (int u = 0; u < 2; ++u)
#pragma unroll 1
          for (int i = 0; i < nks(u); ++i) {
            const SmemDescBase a = make_smem_desc_base(sR(u), 16, 1024);
            const SmemDescBase b = make_smem_desc_base(sCol + 2 * (kt0(u) + i) * kTile, 16, 1024);
#pragma unroll 1
            for (int ks = 0; ks < CN / 16; ++ks) {
              const uint32_t off = (ks / 4) * kTile + (ks % 4) * 32;
              tc_mma_f16(tmem + 128u * (cb0(u) + i), smem_desc_at(a, off), smem_desc_at(b, off), idesc, ks != 0);
            }
          }
        tc_commit(bar_cb);
      }
      const uint32_t idesc_v = make_idesc_f16(128, CP, FMT, 0, 1), idesc_h = make_idesc_f16(128, CP, FMT, 0, 0);
      // None of these loops is unrolled: unrolled, the compiler kept the descriptors of all 40 products of a head across
      // the loop, more than the registers of this warp hold, and every issue waited for a reload from L2 (shared memory
      // leaves L1 nothing): 296 us instead of 174 us for y at 16384 tokens, 80 heads.
#pragma unroll 1
      for (int it = 0; it < n_heads && ok; ++it) {
        const int s = it & 1;
        if (!mbar_wait(full(s), (it >> 1) & 1, p.status, kTimeoutMma)) break;
        const SmemDescBase v = make_smem_desc_base(sV(s), 8192, 1024), hd = make_smem_desc_base(sH(s), 16, 1024);
#pragma unroll 1
        for (int u = 0; u < 2; ++u) {
          if (!mbar_wait(g_full(u), it & 1, p.status, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
#pragma unroll 1
          for (int ks = 0; ks < nks(u) * 8; ++ks)
            tc_mma_f16_ts(tAcc(u), tG(u) + ks * 8, smem_desc_at(v, kt0(u) * kTile + ks * 2048), idesc_v, ks != 0);
          const SmemDescBase r = make_smem_desc_base(sR(u), 16, 1024);
#pragma unroll 1
          for (int ks = 0; ks < CN / 16; ++ks)
            tc_mma_f16(tAcc(u) + 64u, smem_desc_at(r, (ks / 4) * kTile + (ks % 4) * 32),
                       smem_desc_at(hd, (ks / 4) * (kTile / 2) + (ks % 4) * 32), idesc_h, ks != 0);
          tc_commit(acc_full(u));
        }
        if (MODE == 1 && ok) tc_commit(empty(s));  // nothing but the tensor core reads V and H
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kScanRegsCompute));
    const int quarter = warp & 3, chalf = (warp - 4) >> 2;
    const int ctid = threadIdx.x - 128;
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const float* Lg = p.Lt + ((long long)c * p.nh + h_begin) * CQ + ctid;
    const float* dg = p.dtt + ((long long)c * p.nh + h_begin) * CQ + ctid;
    float nL = Lg[0], nd = dg[0];
    // C B^T of this thread's two rows (one per tile) as 16-bit pairs; blocks of 32 columns are taken in turn by the two
    // column halves, so that their causal work is equal.  cb[b]: blocks of tile 0, then of tile 1.
    uint32_t cb[6][16];
    bool ok = mbar_wait(bar_cb, 0, p.status, kTimeoutEpilogue);
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        uint32_t r[32];
        tmem_ld_32x32(tmem + lane_addr + (2 * i + chalf) * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) cb[i][j] = pack2f<FMT>(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
      }
      tc_fence_before();
    }
    auto build_as = [&](int u, const HeadScalars& q, auto split) {
      const int pos = u * 128 + row, rbase = u * 128 + quarter * 32;
      const float Lrow = q.L[pos], drow = MODE == 2 ? q.d[pos] : 1.f;
      const float ref_row = q.ref[pos >> 3], f_row = MODE == 2 ? q.cf[pos] : q.rf[pos];
      const uint64_t f_row2 = pack_f32x2(f_row, f_row);
#pragma unroll
      for (int i = 0; i < 2 * nks(u); ++i) {
        const int b = 2 * i + chalf, col0 = kt0(u) * 128 + b * 32;
        uint32_t pk[16];
        if (MODE == 2 ? col0 < rbase : col0 > rbase) {  // wholly above the diagonal
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = 0u;
        } else {
          const float4 r4 = *reinterpret_cast<const float4*>(&q.ref[col0 >> 3]);
          const float refs[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
          for (int gq = 0; gq < 4; ++gq) {
            const int cg = col0 + gq * 8;
            float f[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t w = cb[2 * cb0(u) + i][gq * 4 + j];
              asm volatile("" : "+r"(w));  // unpack here, not ahead of the loop over the heads: 192 floats spill (174 -> 144 us)
              unpack2<FMT>(w, f[2 * j], f[2 * j + 1]);
            }
            if constexpr (decltype(split)::value) {
              const float e = __expf(MODE == 2 ? refs[gq] - ref_row : ref_row - refs[gq]);
              const float* fc = MODE == 2 ? &q.rf[cg] : &q.cf[cg];
              const float4 c0 = *reinterpret_cast<const float4*>(fc), c1 = *reinterpret_cast<const float4*>(fc + 4);
              const uint64_t cc[4] = {pack_f32x2(c0.x, c0.y), pack_f32x2(c0.z, c0.w), pack_f32x2(c1.x, c1.y), pack_f32x2(c1.z, c1.w)};
              // (CB (e rf_t)) cf_s: t is the row in modes 0 and 1, the column in mode 2
              const float er = MODE == 2 ? e : e * f_row;
              const uint64_t er2 = pack_f32x2(er, er);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint64_t v = pack_f32x2(f[2 * j], f[2 * j + 1]);
                unpack_f32x2(MODE == 2 ? mul_f32x2(mul_f32x2(v, mul_f32x2(er2, cc[j])), f_row2) : mul_f32x2(mul_f32x2(v, er2), cc[j]),
                             f[2 * j], f[2 * j + 1]);
              }
            } else {
              asm volatile("" ::: "memory");  // no loads of later columns ahead of these: registers
#pragma unroll
              for (int j = 0; j < 8; ++j)
                f[j] *= MODE == 2 ? __expf(q.L[cg + j] - Lrow) * drow : __expf(Lrow - q.L[cg + j]) * q.d[cg + j];
            }
            if (col0 == rbase) {  // the diagonal block
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (MODE == 2 ? gq * 8 + j < lane : gq * 8 + j > lane) f[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) pk[gq * 4 + j] = pack2f<FMT>(f[2 * j], f[2 * j + 1]);
          }
        }
        tmem_st_32x16(tG(u) + lane_addr + b * 16, pk);
      }
    };
    auto build = [&](int u, int it) {
      const HeadScalars& q = hs[it % 3];
      if (all_ok(q)) build_as(u, q, std::true_type{});
      else build_as(u, q, std::false_type{});
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(g_full(u));
    };
    auto drain = [&](int u, int it) {
      const int s = it & 1, h = h_begin + it, w = 2 * it + u, e = w % 3;
      if (ok && u == 0 && MODE != 1) ok = mbar_wait(full(s), (it >> 1) & 1, p.status, kTimeoutEpilogue);
      if (ok && MODE != 0) ok = mbar_wait(e_full(e), (w / 3) & 1, p.status, kTimeoutEpilogue);
      if (ok) ok = mbar_wait(acc_full(u), it & 1, p.status, kTimeoutEpilogue);
      const HeadScalars& q = hs[it % 3];
      float d0 = 0.f, d1 = 0.f, d2 = 0.f;
      if (ok) {
        tc_fence_after();
        const int pos = u * 128 + row;
        const float Lrow = q.L[pos];
        // weight of the second product: exp(L_t) for rows t, w_s for rows s
        const float ew = MODE == 2 ? __expf(q.L[CQ - 1] - Lrow) * q.d[pos] : __expf(Lrow);
        const float dh = MODE == 1 ? 0.f : p.D[h];
        const bool still = MODE == 2 && ((q.zero[pos >> 5] >> lane) & 1u) != 0;  // dt = 0: the row gets D dy alone
        uint32_t ra[16], ri[16];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          if ((ch & 1) == 0) {
            tmem_ld_32x16(tAcc(u) + lane_addr + chalf * 32 + ch * 8, ra);
            tmem_ld_32x16(tAcc(u) + lane_addr + 64 + chalf * 32 + ch * 8, ri);
            tmem_ld_wait();
          }
          const uint32_t off = swz(row, chalf * 4 + ch);
          uint4 v4 = make_uint4(0u, 0u, 0u, 0u), e4 = v4;
          if (MODE != 1) v4 = lds128(sV(s) + u * kTile + off);
          if (MODE != 0) e4 = lds128(sE(e) + off);
          const uint32_t vw[4] = {v4.x, v4.y, v4.z, v4.w}, xw[4] = {e4.x, e4.y, e4.z, e4.w};
          uint32_t ow[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float v0 = 0.f, v1 = 0.f, x0 = 0.f, x1 = 0.f;
            if (MODE != 1) unpack2<FMT>(vw[j], v0, v1);
            if (MODE != 0) unpack2<FMT>(xw[j], x0, x1);
            const int k = (ch & 1) * 8 + j * 2;
            const float a0 = __uint_as_float(ra[k]), a1 = __uint_as_float(ra[k + 1]);
            const float i0 = ew * __uint_as_float(ri[k]), i1 = ew * __uint_as_float(ri[k + 1]);
            if (MODE == 1) {
              d0 += x0 * (a0 + i0);
              d1 += x1 * (a1 + i1);
            } else {
              ow[j] = pack2f<FMT>(a0 + i0 + dh * v0, a1 + i1 + dh * v1);
              if (MODE == 2) {
                d0 += v0 * x0 + v1 * x1;
                d1 += i0 * x0 + i1 * x1;
                d2 += a0 * x0 + a1 * x1;
              }
            }
          }
          if (still) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float v0, v1;
              unpack2<FMT>(vw[j], v0, v1);
              ow[j] = pack2f<FMT>(dh * v0, dh * v1);
            }
          }
          if (MODE != 1) sts128(sE(e) + off, ow[0], ow[1], ow[2], ow[3]);
        }
        if (MODE == 1) d0 += d1;
        if (MODE != 0 && chalf == 1) {
          float* sd = sdot + (w % 3) * 384 + row;
          sd[0] = d0;
          if (MODE == 2) {
            sd[128] = d1;
            sd[256] = d2;
          }
        }
        if (MODE != 1) fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (u == 1 && MODE != 1 && lane == 0) mbar_arrive(empty(s));
      }
      // the two warps of these 32 rows meet; the first one's lane 0 stores the rows and returns the buffer
      pair_sync(quarter);
      if (ok && chalf == 0) {
        if (MODE != 0) {
          const long long o = ((long long)c * p.nh + h) * CQ + u * 128 + row;
          const float* sd = sdot + (w % 3) * 384 + row;
          p.red[o] = d0 + sd[0];
          if (MODE == 2) {
            const long long plane = (long long)p.nc * p.nh * CQ;
            p.red[plane + o] = d1 + sd[128];
            p.red[2 * plane + o] = d2 + sd[256];
          }
        }
        if (lane == 0) {
          if (MODE == 1) {
            mbar_arrive(e_empty(e));
          } else {
            tma_store_2d(&tmOut, sE(e) + quarter * 4096, h * CP, c * CQ + u * 128 + quarter * 32);
            tma_store_commit();
            tma_store_wait_read<1>();  // the store of the unit before has read its buffer
            if (MODE == 2 && w > 0) mbar_arrive(e_empty((w - 1) % 3));
          }
        }
      }
    };
    publish<MODE>(hs[0], ctid, nL, nd);
    if (n_heads > 1) {
      nL = Lg[CQ];
      nd = dg[CQ];
    }
    compute_sync(1);  // scalars of the first head are there, and C B^T has been read everywhere: G may overwrite it
    tc_fence_after();
    if (ok) build(0, 0);
    for (int it = 0; it < n_heads; ++it) {
      const bool more = it + 1 < n_heads;
      if (more) {
        publish<MODE>(hs[(it + 1) % 3], ctid, nL, nd);
        if (it + 2 < n_heads) {
          nL = Lg[(it + 2) * CQ];
          nd = dg[(it + 2) * CQ];
        }
      }
      if (ok) build(1, it);
      drain(0, it);
      compute_sync(1);
      if (more && ok) build(0, it + 1);
      drain(1, it);
    }
    if (MODE != 1 && chalf == 0 && lane == 0) tma_store_wait<0>();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ----------------------------------------------------------------------------------------
// State kernel.  grid (nc, G * splits), hp heads in turn.  V [256, 64] of a head (x or dy) is scaled by a factor per row
// IN PLACE in shared memory (rounded to 16 bits as the separate pass did), then serves both products:
//   STATE:  S^T [128 n, 64 p] = R^T V        R = B or C of the chunk, MN-major       -> S [nc, nh, 64, 128] fp32
//   ACC:    acc [256 t, 128 n] += V H        H [64, 128] = entering state or dS, summed over the CTA's heads in
//                                            tensor memory                            -> part [splits, T, G*128] fp32
// ----------------------------------------------------------------------------------------
constexpr int kStateStage = 3 * kTile;  // V, H
template <bool STATE>
constexpr int state_smem() {
  return (STATE ? 4 * kTile : 0) + 2 * kStateStage + 1024 + 256;
}

template <int FMT, bool STATE, bool ACC>
__global__ void __launch_bounds__(320, 1)
ssd_state_kernel(const __grid_constant__ CUtensorMap tmR, const __grid_constant__ CUtensorMap tmV,
                 const __grid_constant__ CUtensorMap tmH, const ScanParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sR = base;  // two 64-column halves of 256 rows
  const uint32_t st0 = base + (STATE ? 4 * kTile : 0);
  auto sV = [&](int s) { return st0 + s * kStateStage; };
  auto sH = [&](int s) { return st0 + s * kStateStage + 2 * kTile; };
  const uint32_t bars = st0 + 2 * kStateStage;
  const uint32_t bar_r = bars;
  auto full = [&](int s) { return bars + 8u + 8u * s; };
  auto ready = [&](int s) { return bars + 24u + 8u * s; };
  auto done = [&](int s) { return bars + 40u + 8u * s; };
  const uint32_t holder = bars + 56u;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x;
  const int hpg = p.nh / p.G, spg = gridDim.y / p.G;
  const int g = blockIdx.y / spg, sp = blockIdx.y % spg;
  const int h_begin = g * hpg + sp * p.hp;
  const int n_heads = min(p.hp, (g + 1) * hpg - h_begin);

  if (warp == 1 && lane == 0) {
    mbar_init(bar_r, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(full(s), 1);
      mbar_init(ready(s), 8);
      mbar_init(done(s), 1);
    }
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(holder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(holder));

  if (warp == 0) {
    if (lane == 0) {
      if (STATE) {
        mbar_expect_tx(bar_r, 4 * kTile);
        for (int k = 0; k < 2; ++k)
          for (int i = 0; i < 2; ++i)
            tma_load_2d(sR + (2 * k + i) * kTile, &tmR, bar_r, g * CN + 64 * k, c * CQ + 128 * i);
      }
      for (int it = 0; it < n_heads; ++it) {
        const int s = it & 1, h = h_begin + it;
        if (!mbar_wait(done(s), ((it >> 1) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(full(s), (2 + (ACC ? 1 : 0)) * kTile);
        for (int i = 0; i < 2; ++i) tma_load_2d(sV(s) + i * kTile, &tmV, full(s), h * CP, c * CQ + 128 * i);
        if (ACC)
          for (int k = 0; k < 2; ++k) tma_load_2d(sH(s) + k * (kTile / 2), &tmH, full(s), 64 * k, (c * p.nh + h) * CP);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = !STATE || mbar_wait(bar_r, 0, p.status, kTimeoutMma);
      const uint32_t idesc_s = make_idesc_f16(128, CP, FMT, 1, 1), idesc_a = make_idesc_f16(128, CN, FMT, 0, 1);
      for (int it = 0; it < n_heads && ok; ++it) {
        const int s = it & 1;
        if (!mbar_wait(ready(s), (it >> 1) & 1, p.status, kTimeoutMma)) break;
        tc_fence_after();
        if (STATE) {
          const SmemDescBase a = make_smem_desc_base(sR, 2 * kTile, 1024), b = make_smem_desc_base(sV(s), 8192, 1024);
#pragma unroll
          for (int ks = 0; ks < CQ / 16; ++ks)
            tc_mma_f16(tmem + 64u * s, smem_desc_at(a, ks * 2048), smem_desc_at(b, ks * 2048), idesc_s, ks != 0);
        }
        if (ACC) {
          const SmemDescBase b = make_smem_desc_base(sH(s), kTile / 2, 1024);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const SmemDescBase a = make_smem_desc_base(sV(s) + i * kTile, 16, 1024);
#pragma unroll
            for (int ks = 0; ks < CP / 16; ++ks)
              tc_mma_f16(tmem + 128u + 128u * i, smem_desc_at(a, ks * 32), smem_desc_at(b, ks * 2048), idesc_a, (it | ks) != 0);
          }
        }
        tc_commit(done(s));
      }
    }
  } else {
    const int quarter = warp & 3, chalf = (warp - 2) >> 2;
    const int ctid = threadIdx.x - 64;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const long long lb = ((long long)c * p.nh + h_begin) * CQ;
    bool ok = true;
    float nL = p.Lt[lb + ctid], nd = p.dtt[lb + ctid], nT = p.Lt[lb + CQ - 1];
    auto scale = [&](int it) {
      const int s = it & 1;
      const float w = p.wmode == 0 ? __expf(nT - nL) * nd : __expf(nL);
      if (it + 1 < n_heads) {
        const long long o = lb + (long long)(it + 1) * CQ;
        nL = p.Lt[o + ctid];
        nd = p.dtt[o + ctid];
        nT = p.Lt[o + CQ - 1];
      }
      if (ok) ok = mbar_wait(full(s), (it >> 1) & 1, p.status, kTimeoutEpilogue);
      if (!ok) return;
#pragma unroll
      for (int ch = 0; ch < 8; ++ch) {
        const uint32_t a = sV(s) + swz(ctid, ch);
        uint4 u = lds128(a);
        uint32_t uw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float v0, v1;
          unpack2<FMT>(uw[j], v0, v1);
          uw[j] = pack2f<FMT>(v0 * w, v1 * w);
        }
        sts128(a, uw[0], uw[1], uw[2], uw[3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ready(s));
    };
    scale(0);
    for (int it = 0; it < n_heads && ok; ++it) {
      const int s = it & 1, h = h_begin + it;
      if (it + 1 < n_heads) scale(it + 1);
      if (STATE) {
        if (ok) ok = mbar_wait(done(s), (it >> 1) & 1, p.status, kTimeoutEpilogue);
        if (!ok) break;
        tc_fence_after();
        uint32_t r[32];
        tmem_ld_32x32(tmem + lane_addr + 64u * s + chalf * 32, r);
        tmem_ld_wait();
        float* out = p.S + (((long long)c * p.nh + h) * CP + chalf * 32) * CN + quarter * 32 + lane;
#pragma unroll
        for (int i = 0; i < 32; ++i) out[i * CN] = __uint_as_float(r[i]);
      }
    }
    if (ACC) {
      const int last = n_heads - 1;
      if (ok && mbar_wait(done(last & 1), (last >> 1) & 1, p.status, kTimeoutEpilogue)) {
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          const long long t = (long long)c * CQ + i * 128 + quarter * 32 + lane;
          float* out = p.part + ((long long)sp * p.T + t) * (p.G * CN) + g * CN + chalf * 64;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            uint32_t r[32];
            tmem_ld_32x32(tmem + lane_addr + 128u + 128u * i + chalf * 64 + k * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<uint4*>(out + k * 32 + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
          }
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ----------------------------------------------------------------------------------------
// dCB.  grid (nc * 3, G * splits): tile pair (t, s) in {(0,0), (1,0), (1,1)}, hp heads in turn.  dy x^T [128, 128] of a
// head (fp32 in tensor memory, two buffers) is weighted by the decay and summed in 64 registers a thread.
// part [splits, nc*G*3, 128, 128] fp32; elements above the diagonal are zeroed by the reduction that follows.
// ----------------------------------------------------------------------------------------
constexpr int kDcbStages = 4;
constexpr int kDcbSmem = kDcbStages * 2 * kTile + 3 * (int)sizeof(HeadScalars) + 1024 + 256;

template <int FMT>
__global__ void __launch_bounds__(320, 1)
ssd_dcb_kernel(const __grid_constant__ CUtensorMap tmDy, const __grid_constant__ CUtensorMap tmX, const ScanParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  auto sA = [&](int s) { return base + s * 2 * kTile; };
  auto sB = [&](int s) { return base + s * 2 * kTile + kTile; };
  const uint32_t scal = base + kDcbStages * 2 * kTile;
  const uint32_t bars = scal + 3 * (uint32_t)sizeof(HeadScalars);
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 32u + 8u * s; };
  auto dg_full = [&](int b) { return bars + 64u + 8u * b; };
  auto dg_empty = [&](int b) { return bars + 80u + 8u * b; };
  const uint32_t holder = bars + 96u;
  HeadScalars* hs = reinterpret_cast<HeadScalars*>(smem_raw + (scal - smem_u32(smem_raw)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x / 3, pair = blockIdx.x % 3;
  const int tt = pair > 0 ? 1 : 0, ts = pair == 2 ? 1 : 0;
  const int hpg = p.nh / p.G, spg = gridDim.y / p.G;
  const int g = blockIdx.y / spg, sp = blockIdx.y % spg;
  const int h_begin = g * hpg + sp * p.hp;
  const int n_heads = min(p.hp, (g + 1) * hpg - h_begin);

  if (warp == 1 && lane == 0) {
    for (int s = 0; s < kDcbStages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(dg_full(b), 1);
      mbar_init(dg_empty(b), 8);
    }
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(holder, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(holder));

  if (warp == 0) {
    if (lane == 0) {
      for (int it = 0; it < n_heads; ++it) {
        const int s = it % kDcbStages, h = h_begin + it;
        if (!mbar_wait(empty(s), ((it / kDcbStages) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(full(s), 2 * kTile);
        tma_load_2d(sA(s), &tmDy, full(s), h * CP, c * CQ + tt * 128);
        tma_load_2d(sB(s), &tmX, full(s), h * CP, c * CQ + ts * 128);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_f16(128, 128, FMT, 0, 0);
      for (int it = 0; it < n_heads; ++it) {
        const int s = it % kDcbStages, b = it & 1;
        if (!mbar_wait(full(s), (it / kDcbStages) & 1, p.status, kTimeoutMma)) break;
        if (!mbar_wait(dg_empty(b), ((it >> 1) & 1) ^ 1u, p.status, kTimeoutMma)) break;
        tc_fence_after();
        const SmemDescBase a = make_smem_desc_base(sA(s), 16, 1024), bb = make_smem_desc_base(sB(s), 16, 1024);
#pragma unroll
        for (int ks = 0; ks < CP / 16; ++ks)
          tc_mma_f16(tmem + 128u * b, smem_desc_at(a, ks * 32), smem_desc_at(bb, ks * 32), idesc, ks != 0);
        tc_commit(empty(s));
        tc_commit(dg_full(b));
      }
    }
  } else {
    const int quarter = warp & 3, chalf = (warp - 2) >> 2;
    const int ctid = threadIdx.x - 64;
    const int row = quarter * 32 + lane;
    const int pos = tt * 128 + row, col0 = ts * 128 + chalf * 64;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const float* Lg = p.Lt + ((long long)c * p.nh + h_begin) * CQ + ctid;
    const float* dg = p.dtt + ((long long)c * p.nh + h_begin) * CQ + ctid;
    float nL = Lg[0], nd = dg[0];
    uint64_t acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0ull;
    bool ok = true;
    for (int it = 0; it < n_heads; ++it) {
      const int b = it & 1;
      HeadScalars& q = hs[it % 3];
      publish<3>(q, ctid, nL, nd);
      if (it + 1 < n_heads) {
        nL = Lg[(it + 1) * CQ];
        nd = dg[(it + 1) * CQ];
      }
      compute_sync(1);
      if (ok) ok = mbar_wait(dg_full(b), (it >> 1) & 1, p.status, kTimeoutEpilogue);
      if (!ok) continue;
      tc_fence_after();
      const float Lrow = q.L[pos];
      const bool split = all_ok(q);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        uint32_t r[32];
        tmem_ld_32x32(tmem + 128u * b + lane_addr + chalf * 64 + k * 32, r);
        tmem_ld_wait();
        if (k == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dg_empty(b));
        }
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          const int cg = col0 + k * 32 + gq * 8;
          uint64_t* ac = acc + k * 16 + gq * 4;
          if (split) {
            const float e = __expf(Lrow - q.ref[cg >> 3]);
            const uint64_t e2 = pack_f32x2(e, e);
            const float4 c0 = *reinterpret_cast<const float4*>(&q.cf[cg]), c1 = *reinterpret_cast<const float4*>(&q.cf[cg + 4]);
            const uint64_t cf[4] = {pack_f32x2(c0.x, c0.y), pack_f32x2(c0.z, c0.w), pack_f32x2(c1.x, c1.y), pack_f32x2(c1.z, c1.w)};
#pragma unroll
            for (int j = 0; j < 4; ++j)
              ac[j] = fma_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(r[gq * 8 + 2 * j]), __uint_as_float(r[gq * 8 + 2 * j + 1])), e2),
                                cf[j], ac[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float w0 = __expf(Lrow - q.L[cg + 2 * j]) * q.d[cg + 2 * j];
              const float w1 = __expf(Lrow - q.L[cg + 2 * j + 1]) * q.d[cg + 2 * j + 1];
              ac[j] = fma_f32x2(pack_f32x2(__uint_as_float(r[gq * 8 + 2 * j]), __uint_as_float(r[gq * 8 + 2 * j + 1])),
                                pack_f32x2(w0, w1), ac[j]);
            }
          }
        }
      }
    }
    if (ok) {
      float* out = p.part + (((long long)sp * p.nc + c) * p.G + g) * (3 * 128 * 128) + (pair * 128 + row) * 128 + chalf * 64;
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        float4 v;
        unpack_f32x2(acc[j], v.x, v.y);
        unpack_f32x2(acc[j + 1], v.z, v.w);
        *reinterpret_cast<float4*>(out + 2 * j) = v;
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// dCB in 16 bits, [nc*G, 256, 256], zero above the diagonal: the sum of the head splits' partial tiles.
// grid nc*G*32, block 256: eight rows per CTA, eight columns per thread.
template <int FMT>
__global__ void __launch_bounds__(256) ssd_dcb_reduce_kernel(const float* __restrict__ part, uint4* __restrict__ out, int splits,
                                                             long long tiles) {
  const int m = blockIdx.x >> 5;
  const int t = (blockIdx.x & 31) * 8 + (threadIdx.x >> 5), s0 = (threadIdx.x & 31) * 8;
  float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (s0 <= t) {
    const int pair = t < 128 ? 0 : (s0 < 128 ? 1 : 2);
    const float* src = part + (long long)m * 49152 + (pair * 128 + (t & 127)) * 128 + (s0 & 127);
    for (int k = 0; k < splits; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
      f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
      f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
      src += tiles * 49152;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (s0 + j > t) f[j] = 0.f;
  }
  out[((long long)m * CQ + t) * 32 + (threadIdx.x & 31)] = make_uint4(pack2f<FMT>(f[0], f[1]), pack2f<FMT>(f[2], f[3]),
                                                                      pack2f<FMT>(f[4], f[5]), pack2f<FMT>(f[6], f[7]));
}

// out (16-bit) = sum of `splits` fp32 partials of n elements + add (fp32); eight elements per thread.
template <int FMT>
__global__ void __launch_bounds__(256) ssd_sum_kernel(const float* __restrict__ part, const float* __restrict__ add,
                                                      uint4* __restrict__ out, int splits, long long n) {
  const long long i = (blockIdx.x * 256LL + threadIdx.x) * 8;
  if (i >= n) return;
  float4 a = *reinterpret_cast<const float4*>(add + i), b = *reinterpret_cast<const float4*>(add + i + 4);
  for (int k = 0; k < splits; ++k) {
    const float4 u = *reinterpret_cast<const float4*>(part + k * n + i), v = *reinterpret_cast<const float4*>(part + k * n + i + 4);
    a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
    b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
  }
  out[i >> 3] = make_uint4(pack2f<FMT>(a.x, a.y), pack2f<FMT>(a.z, a.w), pack2f<FMT>(b.x, b.y), pack2f<FMT>(b.z, b.w));
}

// ----------------------------------------------------------------------------------------
// Decay bookkeeping: a warp per head, eight positions per lane.  grid (nc, ceil(nh / 8)), block 256.
// ----------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) ssd_decay_kernel(const float* __restrict__ dt, const float* __restrict__ A,
                                                        float* __restrict__ Lt, float* __restrict__ dtt,
                                                        float* __restrict__ Ltot, int nh) {
  __shared__ float sd[8][CQ + 4];
  const int c = blockIdx.x, h0 = blockIdx.y * 8;
  for (int i = threadIdx.x; i < CQ * 8; i += 256) {
    const int t = i >> 3, h = i & 7;
    sd[h][t] = h0 + h < nh ? dt[((long long)c * CQ + t) * nh + h0 + h] : 0.f;
  }
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = h0 + w;
  if (h >= nh) return;
  const float a = A[h];
  float d[8], s[8], run = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    d[j] = sd[w][lane * 8 + j];
    run += d[j] * a;
    s[j] = run;
  }
  float inc = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  float before = __shfl_up_sync(0xffffffffu, inc, 1);
  if (lane == 0) before = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] += before;
  const long long o = ((long long)c * nh + h) * CQ + lane * 8;
  *reinterpret_cast<float4*>(Lt + o) = make_float4(s[0], s[1], s[2], s[3]);
  *reinterpret_cast<float4*>(Lt + o + 4) = make_float4(s[4], s[5], s[6], s[7]);
  *reinterpret_cast<float4*>(dtt + o) = make_float4(d[0], d[1], d[2], d[3]);
  *reinterpret_cast<float4*>(dtt + o + 4) = make_float4(d[4], d[5], d[6], d[7]);
  if (lane == 31) Ltot[(long long)c * nh + h] = s[7];
}

// Gradients through the decay.  yd = dy . (y - D x), dww = w x.(B dS^T), col = x.(G^T dy), dyx = dy . x per (chunk, head,
// position).  dL = yd - dww - col (+ dLtot and the sum of dww at the last position); through L = cumsum(dt A) that is a
// reverse cumulative sum da; ddt = (dww + col) / dt + da A; partial dA = sum da dt and dD = sum dyx per (chunk, head).  Where dt
// is 0, dww and col come without it (see publish): they are the derivative themselves and have no part in dL.
__global__ void __launch_bounds__(256) ssd_decay_bwd_kernel(const float* __restrict__ yd, const float* __restrict__ red,
                                                            const float* __restrict__ dtt, const float* __restrict__ A,
                                                            const float* __restrict__ dLtot, float* __restrict__ ddt,
                                                            float* __restrict__ sums, int nc, int nh) {
  __shared__ float sd[8][CQ + 4];
  const int c = blockIdx.x, h0 = blockIdx.y * 8;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = h0 + w;
  const long long plane = (long long)nc * nh * CQ;
  if (h < nh) {
    const long long o = ((long long)c * nh + h) * CQ + lane * 8;
    auto ld = [](const float* q, float (&f)[8]) {
      const float4 u = *reinterpret_cast<const float4*>(q), v = *reinterpret_cast<const float4*>(q + 4);
      f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w;
      f[4] = v.x; f[5] = v.y; f[6] = v.z; f[7] = v.w;
    };
    float y[8], k[8], ww[8], co[8], d[8];
    ld(yd + o, y);
    ld(red + o, k);
    ld(red + plane + o, ww);
    ld(red + 2 * plane + o, co);
    ld(dtt + o, d);
    float sw = 0.f, sk = 0.f, direct[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      direct[j] = ww[j] + co[j];
      if (d[j] == 0.f) ww[j] = co[j] = 0.f;
      else direct[j] /= d[j];
      sw += ww[j];
      sk += k[j];
    }
    sw = warp_sum(sw);
    sk = warp_sum(sk);
    const float a = A[h];
    float dl[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dl[j] = y[j] - ww[j] - co[j];
    if (lane == 31) dl[7] += dLtot[(long long)c * nh + h] + sw;
    float run = 0.f;
#pragma unroll
    for (int j = 7; j >= 0; --j) {
      run += dl[j];
      dl[j] = run;
    }
    float inc = run;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
      const float v = __shfl_down_sync(0xffffffffu, inc, q);
      if (lane + q < 32) inc += v;
    }
    float after = __shfl_down_sync(0xffffffffu, inc, 1);
    if (lane == 31) after = 0.f;
    float sa = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float da = dl[j] + after;
      sa += da * d[j];
      sd[w][lane * 8 + j] = direct[j] + da * a;
    }
    sa = warp_sum(sa);
    if (lane == 0) {
      sums[(long long)c * nh + h] = sa;
      sums[(long long)nc * nh + (long long)c * nh + h] = sk;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < CQ * 8; i += 256) {
    const int t = i >> 3, k = i & 7;
    if (h0 + k < nh) ddt[((long long)c * CQ + t) * nh + h0 + k] = sd[k][t];
  }
}

}  // namespace ssdf
}  // namespace fmsb

using namespace fmsb;
using namespace fmsb::ssdf;

// Heads per CTA: the split of a group's heads for which the machine (148 SMs, one CTA each) finishes first, a CTA
// costing its heads plus about two heads' worth of prologue and drain.
static int pick_heads(long long tiles, int hpg) {
  long long best = -1;
  int hp = hpg;
  for (int spg = 1; spg <= hpg; ++spg) {
    const int n = (hpg + spg - 1) / spg;
    if ((hpg + n - 1) / n != spg) continue;
    const long long cost = (tiles * spg + 147) / 148 * (n + 2);
    if (best < 0 || cost < best) { best = cost; hp = n; }
  }
  return hp;
}

// kind 0: scan and 1: state kernel (one CTA per chunk, group and split), 2: dCB (three).  Returns heads per CTA.
extern "C" int fmsb_ssdf_heads(int kind, int nc, int nh, int G) {
  if (nc <= 0 || G <= 0 || nh % G) return 1;
  return pick_heads((long long)nc * G * (kind == 2 ? 3 : 1), nh / G);
}

static int map_rows(CUtensorMap* m, const void* p, long long rows, long long cols, long long ld, int box_rows) {
  return fmsb_host::make_tmap_2d_16b(m, p, rows, cols, ld, box_rows, 64);
}

template <typename K>
static int set_smem(K kern, int bytes) {
  return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// The register split of the scan kernel draws on what the block was launched with: a build that gave the kernel fewer
// registers per thread would wait for them without end, so it is refused here.
template <typename K>
static int scan_regs(K kern) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kern);
  if (e != cudaSuccess) return (int)e;
  return a.numRegs * kScanThreads >= 128 * kScanRegsMain + 256 * kScanRegsCompute ? 0 : -3;
}

// mode 0: out = y (v = x, r = C, col = B, hst = entering states); mode 1: red = dy . y-terms (e = dy);
// mode 2: out = dx and red (v = dy, r = B, col = C, hst = dS, e = x).  v, e, out [nc*256, nh*64] dense; r, col rows of
// G*128 with leading dimensions ldr / ldc; hst [nc*nh*64, 128].
extern "C" int fmsb_ssdf_scan(int mode, const void* r, long long ldr, const void* col, long long ldc, const void* v,
                              const void* hst, const void* e, void* out, const float* Lt, const float* dtt, const float* D,
                              float* red, int nc, int nh, int G, int hp, int fmt, int* status, cudaStream_t stream) {
  if (nc <= 0) return 0;
  if (nh % G || hp <= 0 || (ldr % 8) || (ldc % 8) || fmt < 0 || fmt > 1 || mode < 0 || mode > 2) return -2;
  const long long T = (long long)nc * CQ;
  CUtensorMap tr, tc, tv, th, te, to;
  int rc;
  if ((rc = map_rows(&tr, r, T, (long long)G * CN, ldr, 128))) return rc;
  if ((rc = map_rows(&tc, col, T, (long long)G * CN, ldc, 128))) return rc;
  if ((rc = map_rows(&tv, v, T, (long long)nh * CP, (long long)nh * CP, 128))) return rc;
  if ((rc = map_rows(&th, hst, (long long)nc * nh * CP, CN, CN, 64))) return rc;
  te = tv;
  to = tv;
  if (mode != 0 && (rc = map_rows(&te, e, T, (long long)nh * CP, (long long)nh * CP, 128))) return rc;
  if (mode != 1 && (rc = map_rows(&to, out, T, (long long)nh * CP, (long long)nh * CP, 32))) return rc;
  ScanParams p{};
  p.nc = nc; p.nh = nh; p.G = G; p.hp = hp; p.Lt = Lt; p.dtt = dtt; p.D = D; p.red = red; p.T = (int)T; p.status = status;
  const int hpg = nh / G;
  const dim3 grid(nc, G * ((hpg + hp - 1) / hp));
#define FMSB_SCAN(MM, FF)                                                                              \
  do {                                                                                                 \
    static bool cfg = false;                                                                           \
    if (!cfg) {                                                                                        \
      if ((rc = set_smem(ssd_scan_kernel<MM, FF>, kScanSmem))) return rc;                              \
      if ((rc = scan_regs(ssd_scan_kernel<MM, FF>))) return rc;                                        \
      cfg = true;                                                                                      \
    }                                                                                                  \
    ssd_scan_kernel<MM, FF><<<grid, kScanThreads, kScanSmem, stream>>>(tr, tc, tv, th, te, to, p);              \
  } while (0)
  if (fmt == 1) { if (mode == 0) FMSB_SCAN(0, 1); else if (mode == 1) FMSB_SCAN(1, 1); else FMSB_SCAN(2, 1); }
  else { if (mode == 0) FMSB_SCAN(0, 0); else if (mode == 1) FMSB_SCAN(1, 0); else FMSB_SCAN(2, 0); }
#undef FMSB_SCAN
  return (int)cudaGetLastError();
}

// S (may be null) [nc, nh, 64, 128] = (v w)^T r; part (may be null) [splits, T, G*128] = sum over heads of (v w) hst.
extern "C" int fmsb_ssdf_state(const void* r, long long ldr, const void* v, const void* hst, const float* Lt,
                               const float* dtt, float* S, float* part, int wmode, int nc, int nh, int G, int hp, int fmt,
                               int* status, cudaStream_t stream) {
  if (nc <= 0) return 0;
  if (nh % G || hp <= 0 || fmt < 0 || fmt > 1 || (S == nullptr && part == nullptr) || (S != nullptr && (ldr % 8))) return -2;
  const long long T = (long long)nc * CQ;
  CUtensorMap tr, tv, th;
  int rc;
  if ((rc = map_rows(&tv, v, T, (long long)nh * CP, (long long)nh * CP, 128))) return rc;
  tr = tv;
  th = tv;
  if (S != nullptr && (rc = map_rows(&tr, r, T, (long long)G * CN, ldr, 128))) return rc;
  if (part != nullptr && (rc = map_rows(&th, hst, (long long)nc * nh * CP, CN, CN, 64))) return rc;
  ScanParams p{};
  p.nc = nc; p.nh = nh; p.G = G; p.hp = hp; p.Lt = Lt; p.dtt = dtt; p.S = S; p.part = part; p.wmode = wmode; p.T = (int)T;
  p.status = status;
  const int hpg = nh / G;
  const dim3 grid(nc, G * ((hpg + hp - 1) / hp));
#define FMSB_STATE(FF, SS, AA)                                                                   \
  do {                                                                                           \
    static bool cfg = false;                                                                     \
    if (!cfg) {                                                                                  \
      if ((rc = set_smem(ssd_state_kernel<FF, SS, AA>, state_smem<SS>()))) return rc;            \
      cfg = true;                                                                                \
    }                                                                                            \
    ssd_state_kernel<FF, SS, AA><<<grid, 320, state_smem<SS>(), stream>>>(tr, tv, th, p);        \
  } while (0)
  if (fmt == 1) {
    if (S && part) FMSB_STATE(1, true, true); else if (S) FMSB_STATE(1, true, false); else FMSB_STATE(1, false, true);
  } else {
    if (S && part) FMSB_STATE(0, true, true); else if (S) FMSB_STATE(0, true, false); else FMSB_STATE(0, false, true);
  }
#undef FMSB_STATE
  return (int)cudaGetLastError();
}

// dcb [nc*G, 256, 256] 16-bit; part: scratch of splits * nc * G * 3 * 128 * 128 floats.
extern "C" int fmsb_ssdf_dcb(const void* dy, const void* x, const float* Lt, const float* dtt, float* part, void* dcb, int nc,
                             int nh, int G, int hp, int fmt, int* status, cudaStream_t stream) {
  if (nc <= 0) return 0;
  if (nh % G || hp <= 0 || fmt < 0 || fmt > 1) return -2;
  const long long T = (long long)nc * CQ;
  CUtensorMap td, tx;
  int rc;
  if ((rc = map_rows(&td, dy, T, (long long)nh * CP, (long long)nh * CP, 128))) return rc;
  if ((rc = map_rows(&tx, x, T, (long long)nh * CP, (long long)nh * CP, 128))) return rc;
  ScanParams p{};
  p.nc = nc; p.nh = nh; p.G = G; p.hp = hp; p.Lt = Lt; p.dtt = dtt; p.part = part; p.T = (int)T; p.status = status;
  const int spg = (nh / G + hp - 1) / hp;
  const dim3 grid(nc * 3, G * spg);
#define FMSB_DCB(FF)                                                                                              \
  do {                                                                                                            \
    static bool cfg = false;                                                                                      \
    if (!cfg) {                                                                                                   \
      if ((rc = set_smem(ssd_dcb_kernel<FF>, kDcbSmem))) return rc;                                               \
      cfg = true;                                                                                                 \
    }                                                                                                             \
    ssd_dcb_kernel<FF><<<grid, 320, kDcbSmem, stream>>>(td, tx, p);                                               \
    ssd_dcb_reduce_kernel<FF><<<nc * G * 32, 256, 0, stream>>>(part, (uint4*)dcb, spg, (long long)nc * G);        \
  } while (0)
  if (fmt == 1) FMSB_DCB(1);
  else FMSB_DCB(0);
#undef FMSB_DCB
  return (int)cudaGetLastError();
}

extern "C" int fmsb_ssdf_sum(const float* part, const float* add, void* out, int splits, long long n, int fmt,
                             cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8 || fmt < 0 || fmt > 1) return -2;
  const unsigned blocks = (unsigned)((n / 8 + 255) / 256);
  if (fmt == 1) ssd_sum_kernel<1><<<blocks, 256, 0, stream>>>(part, add, (uint4*)out, splits, n);
  else ssd_sum_kernel<0><<<blocks, 256, 0, stream>>>(part, add, (uint4*)out, splits, n);
  return (int)cudaGetLastError();
}

extern "C" int fmsb_ssdf_decay(const float* dt, const float* A, float* Lt, float* dtt, float* Ltot, int nc, int nh,
                               cudaStream_t stream) {
  if (nc <= 0 || nh <= 0) return 0;
  ssd_decay_kernel<<<dim3(nc, (nh + 7) / 8), 256, 0, stream>>>(dt, A, Lt, dtt, Ltot, nh);
  return (int)cudaGetLastError();
}

extern "C" int fmsb_ssdf_decay_bwd(const float* yd, const float* red, const float* dtt, const float* A, const float* dLtot,
                                   float* ddt, float* sums, int nc, int nh, cudaStream_t stream) {
  if (nc <= 0 || nh <= 0) return 0;
  ssd_decay_bwd_kernel<<<dim3(nc, (nh + 7) / 8), 256, 0, stream>>>(yd, red, dtt, A, dLtot, ddt, sums, nc, nh);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------
// The launches of a whole forward and of a whole backward in one call each: from Python every launch costs the host some
// 10 us (allocation, argument conversion, tensor maps apart), and at a few thousand tokens the kernels are shorter than that.
// 1024 tokens, 48 heads, forward: 65 -> 44 us a pass; 4352 tokens, forward and backward: 406 -> 299 us.
// ----------------------------------------------------------------------------------------
extern "C" int fmsb_ssd_state_fwd(const float*, const float*, const float*, void*, float*, int, int, int, int, cudaStream_t);
extern "C" int fmsb_ssd_state_bwd(const float*, const float*, const float*, const void*, void*, float*, float*, int, int, int, int,
                                  cudaStream_t);
extern "C" int fmsb_batched_gemm(const void* A, long long lda, long long a_rows, long long a_cols, const void* B, long long ldb,
                                 long long b_rows, long long b_cols, int K, int a_mn, int b_mn, void* D, long long ldd,
                                 int d_fp32, const void* C, long long ldc, float alpha, float beta, int M, int N, int fmt,
                                 int bn, const int* desc, int* status, cudaStream_t stream);

namespace {
// Carves 256-byte aligned pieces out of a workspace; with a null base it only counts.
struct Carver {
  char* base;
  size_t used = 0;
  explicit Carver(void* b) : base((char*)b) {}
  template <typename T>
  T* take(size_t n) {
    T* p = base == nullptr ? nullptr : reinterpret_cast<T*>(base + used);
    used += (n * sizeof(T) + 255) / 256 * 256;
    return p;
  }
};
struct FwdWs {
  float *Lt, *dtt, *Ltot, *S;
  FwdWs(Carver& c, size_t nc, size_t nh)
      : Lt(c.take<float>(nc * nh * CQ)), dtt(c.take<float>(nc * nh * CQ)), Ltot(c.take<float>(nc * nh)),
        S(c.take<float>(nc * nh * CP * CN)) {}
};
struct BwdWs {
  float *Lt, *dtt, *Ltot, *ydot, *dhp, *partC, *partB, *dLtot, *red, *dcbPart, *gC, *gB;
  uint16_t *dS, *dcb;
  int hp1, sp1, hp2, sp2;
  BwdWs(Carver& c, size_t nc, size_t nh, size_t G) {
    const int hpg = (int)(nh / G);
    hp1 = pick_heads((long long)(nc * G), hpg);
    hp2 = pick_heads((long long)(nc * G * 3), hpg);
    sp1 = (hpg + hp1 - 1) / hp1;
    sp2 = (hpg + hp2 - 1) / hp2;
    const size_t rows = nc * CQ * G * CN;
    Lt = c.take<float>(nc * nh * CQ); dtt = c.take<float>(nc * nh * CQ); Ltot = c.take<float>(nc * nh);
    ydot = c.take<float>(nc * nh * CQ); red = c.take<float>(3 * nc * nh * CQ); dLtot = c.take<float>(nc * nh);
    dhp = c.take<float>(nc * nh * CP * CN); dS = c.take<uint16_t>(nc * nh * CP * CN);
    partC = c.take<float>(sp1 * rows); partB = c.take<float>(sp1 * rows);
    dcbPart = c.take<float>((size_t)sp2 * nc * G * 3 * 128 * 128); dcb = c.take<uint16_t>(nc * G * CQ * CQ);
    gC = c.take<float>(rows); gB = c.take<float>(rows);
  }
};
}  // namespace

// bytes of the workspace of fmsb_ssdf_forward (backward = 0) / fmsb_ssdf_backward (1)
extern "C" long long fmsb_ssdf_workspace(int backward, int nc, int nh, int G) {
  if (nc <= 0 || nh <= 0 || G <= 0 || nh % G) return 0;
  Carver c(nullptr);
  if (backward) BwdWs(c, nc, nh, G);
  else FwdWs(c, nc, nh);
  return (long long)c.used;
}

// x, y [nc*256, nh*64]; dt [nc*256, nh] fp32; A, D [nh] fp32; B, C rows of G*128 (ldb, ldc); h0 (may be null), hT
// [nh, 64, 128] fp32; hprev [nc*nh*64, 128].  y null: the states only.
extern "C" int fmsb_ssdf_forward(const void* x, const float* dt, const float* A, const void* B, long long ldb, const void* C,
                                 long long ldc, const float* D, const float* h0, void* y, float* hT, void* hprev, void* ws,
                                 int nc, int nh, int G, int fmt, int* status, cudaStream_t stream) {
  if (nc <= 0) return 0;
  if (ws == nullptr || G <= 0 || nh % G) return -2;
  Carver c(ws);
  FwdWs w(c, nc, nh);
  const int hp = pick_heads((long long)nc * G, nh / G);
  int rc;
  if ((rc = fmsb_ssdf_decay(dt, A, w.Lt, w.dtt, w.Ltot, nc, nh, stream))) return rc;
  if ((rc = fmsb_ssdf_state(B, ldb, x, nullptr, w.Lt, w.dtt, w.S, nullptr, 0, nc, nh, G, hp, fmt, status, stream))) return rc;
  if ((rc = fmsb_ssd_state_fwd(w.S, w.Ltot, h0, hprev, hT, nc, nh, CP * CN, fmt, stream))) return rc;
  if (y == nullptr) return 0;
  return fmsb_ssdf_scan(0, C, ldc, B, ldb, x, hprev, nullptr, y, w.Lt, w.dtt, D, nullptr, nc, nh, G, hp, fmt, status, stream);
}

// dx [nc*256, nh*64], dB, dC [nc*256, G*128] 16-bit; ddt [nc*256, nh], sums [2, nc, nh] (partial dA, dD), dh0 (may be null)
// fp32; dhT may be null.
extern "C" int fmsb_ssdf_backward(const void* x, const void* dy, const float* dt, const float* A, const void* B, long long ldb,
                                  const void* C, long long ldc, const float* D, const void* hprev, const float* dhT, void* dx,
                                  float* ddt, void* dB, void* dC, float* sums, float* dh0, void* ws, int nc, int nh, int G,
                                  int fmt, int* status, cudaStream_t stream) {
  if (nc <= 0) return 0;
  if (ws == nullptr || G <= 0 || nh % G) return -2;
  Carver c(ws);
  BwdWs w(c, nc, nh, G);
  const long long T = (long long)nc * CQ, gn = (long long)G * CN;
  int rc;
  if ((rc = fmsb_ssdf_decay(dt, A, w.Lt, w.dtt, w.Ltot, nc, nh, stream))) return rc;
  if ((rc = fmsb_ssdf_scan(1, C, ldc, B, ldb, x, hprev, dy, nullptr, w.Lt, w.dtt, nullptr, w.ydot, nc, nh, G, w.hp1, fmt,
                           status, stream))) return rc;
  if ((rc = fmsb_ssdf_state(C, ldc, dy, hprev, w.Lt, w.dtt, w.dhp, w.partC, 1, nc, nh, G, w.hp1, fmt, status, stream))) return rc;
  if ((rc = (int)cudaMemsetAsync(w.dLtot, 0, sizeof(float) * nc * nh, stream))) return rc;
  if ((rc = fmsb_ssd_state_bwd(w.dhp, dhT, w.Ltot, hprev, w.dS, dh0, w.dLtot, nc, nh, CP * CN, fmt, stream))) return rc;
  if ((rc = fmsb_ssdf_scan(2, B, ldb, C, ldc, dy, w.dS, x, dx, w.Lt, w.dtt, D, w.red, nc, nh, G, w.hp1, fmt, status, stream))) return rc;
  if ((rc = fmsb_ssdf_state(B, ldb, x, w.dS, w.Lt, w.dtt, nullptr, w.partB, 0, nc, nh, G, w.hp1, fmt, status, stream))) return rc;
  if ((rc = fmsb_ssdf_dcb(dy, x, w.Lt, w.dtt, w.dcbPart, w.dcb, nc, nh, G, w.hp2, fmt, status, stream))) return rc;
  const int desc[13] = {nc * G, G, G * CQ, CQ, 0, 1, CQ, 0, CN, 1, CQ, 0, CN};
  for (int k = 0; k < 2; ++k) {  // dC = dCB B + ..., dB = dCB^T C + ...
    if ((rc = fmsb_batched_gemm(w.dcb, CQ, T * G, CQ, k == 0 ? B : C, k == 0 ? ldb : ldc, T, gn, CQ, k, 1, k == 0 ? w.gC : w.gB,
                                gn, 1, nullptr, 0, 1.f, 0.f, CQ, CN, fmt, 128, desc, status, stream))) return rc;
    if ((rc = fmsb_ssdf_sum(k == 0 ? w.partC : w.partB, k == 0 ? w.gC : w.gB, k == 0 ? dC : dB, w.sp1, T * gn, fmt, stream))) return rc;
  }
  return fmsb_ssdf_decay_bwd(w.ydot, w.red, w.dtt, A, w.dLtot, ddt, sums, nc, nh, stream);
}
