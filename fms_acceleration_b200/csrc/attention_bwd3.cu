// Attention backward, full-width issue order.  Replaces the backward half of flash_attn_varlen_func as used by the reference's
// padding-free plugin (fms_acceleration_aadp/flash_attn.py:108-199).
//
// What the timeline trace of an earlier half-tile design (128x64 products) showed: the single MMA-issuing thread, not the exponentials,
// was the critical path, because a 128x64x16 product costs almost as much issue/operand time as a 128x128x16 one.
// Here every product is 128 wide and the element-wise work is split into two stages that each overlap a pair of
// products:
//
//   dK/dV kernel (fixed key tile; K and V rows are the M side, queries are streamed)
//     MMA order      S^T(j)  dP^T(j) | dV(j)  S^T(j+1) | dK(j)  dP^T(j+1) | dV(j+1) ...
//     compute order            A(j): P^T = exp2(S^T..) -> packed over S^T      (needs S^T(j))
//                              B(j): dS^T = P^T o (dP^T - delta) -> over dP^T  (needs dP^T(j))
//     dV(j) waits for A(j), dK(j) for B(j); A(j+1) runs while dK(j), dP^T(j+1) execute.
//   dQ kernel (fixed query tile; keys are streamed)
//     MMA order      S(j) dP(j) | S(j+1) dP(j+1) | dQ(j) | S(j+2) dP(j+2) | dQ(j+1) ...
//     compute order  load S(j) (then S(j+1) may overwrite it), P in registers, B(j): dS over dP(j)
//     dP has two buffers: with one, dP(j+1) waited for dQ(j), which waits for B(j), and every block was that chain.
//     The second one takes the room that Q and dO had in tensor memory as A operands; they are read from shared memory.
//     V is released by dP(j), K by dQ(j), so half of the next loads start a product earlier.
//
// Tensor memory (512 columns): dK/dV: S^T 128 | dP^T 128 | dV D | dK D.   dQ: S 128 | dP 2 x 128 | dQ D.
// P is kept as packed 16-bit between the stages (it is the operand of dV in that precision anyway).
// T = 16384 packed, 32/8 heads, d = 128: dQ 919 -> 874 us, dK/dV 1050 -> 886 us (heads fastest in the grids, fp32 pairs),
// then 842 and 884 us with sixteen compute warps instead of eight;
// T = 1500, d = 64: dQ 29.4 -> 21.2 us.
// Warp roles (576 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2-17 compute; a compute warp owns lane
// quarter `warp % 4` and 32 of the 128 columns.  Every wait is bounded.
#include "common.cuh"

namespace fmsb {

constexpr int B3_T = 128;  // tile edge (queries and keys)
constexpr int B3_CW = 16;   // compute warps: four per scheduler, 32 of the 128 columns each (eight of 64 left latency exposed)
constexpr int B3_THREADS = 64 + 32 * B3_CW;

struct AttnBwd3Params {
  int T, nh, nkv, d;
  float scale;
  const int* doc_start;
  const int* doc_end;
  const float* lse;    // [nh, T]
  const float* delta;  // [nh, T]
  void* dq;
  long long lddq;
  void* dk;
  long long lddk;
  void* dv;
  long long lddv;
  int fmt;
  int* status;
};

template <int D>
struct AttnBwd3Cfg {
  static constexpr int kTileBytes = 128 * D * 2;
  static constexpr int kHalfBytes = 128 * 64 * 2;
  static constexpr int kScalarBytes = 2 * 3 * 128 * 4;
  static constexpr int kSmemBytes = 6 * kTileBytes + kScalarBytes + 1024 + 256;
};

__device__ __forceinline__ uint32_t b3_pack2(float a, float b, int fmt) {
  return fmt == 1 ? pack_bf16x2(a, b) : pack_f16x2(a, b);
}
__device__ __forceinline__ void b3_unpack2(uint32_t w, int fmt, float& a, float& b) {
  if (fmt == 1) {
    a = __uint_as_float(w << 16);
    b = __uint_as_float(w & 0xffff0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    a = f.x;
    b = f.y;
  }
}
template <int NC>
__device__ __forceinline__ void b3_store_row_chunk(uint16_t* dst, const uint32_t (&r)[NC], float mul, int fmt) {
#pragma unroll
  for (int i = 0; i < NC; i += 8) {
    uint4 u;
    u.x = b3_pack2(__uint_as_float(r[i]) * mul, __uint_as_float(r[i + 1]) * mul, fmt);
    u.y = b3_pack2(__uint_as_float(r[i + 2]) * mul, __uint_as_float(r[i + 3]) * mul, fmt);
    u.z = b3_pack2(__uint_as_float(r[i + 4]) * mul, __uint_as_float(r[i + 5]) * mul, fmt);
    u.w = b3_pack2(__uint_as_float(r[i + 6]) * mul, __uint_as_float(r[i + 7]) * mul, fmt);
    *reinterpret_cast<uint4*>(dst + i) = u;
  }
}
// Optional timeline trace (compile with -DFMSB_TRACE): one CTA of the dQ kernel records clock64() at the hand-off
// points of its MMA issuer and of one compute thread; read back with fmsb_attn_trace3_read.
#ifdef FMSB_TRACE
__device__ long long g_trace3[8192];
#define FMSB_TRACE3(cond, slot) do { if ((cond) && (slot) < 8192) g_trace3[(slot)] = clock64(); } while (0)
#else
#define FMSB_TRACE3(cond, slot) do { } while (0)
#endif

__device__ __forceinline__ void b3_compute_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// Column of K-step `ks` (16 elements = 8 packed columns) of a packed 128-element row: the warp of columns 32 q .. 32 q + 31
// packs into columns 32 q .. 32 q + 15 (each overwrites only what it has read).
__device__ __forceinline__ uint32_t b3_pcol(int ks) { return static_cast<uint32_t>((ks >> 1) * 32 + (ks & 1) * 8); }

// This warp's quarter of an accumulator row (D / 4 columns from `col`), multiplied, to global memory.
template <int D, int FMT>
__device__ __forceinline__ void b3_store_quarter(uint16_t* dst, uint32_t taddr, float mul, bool on) {
  if constexpr (D == 128) {
    uint32_t r[32];
    tmem_ld_32x32(taddr, r);
    tmem_ld_wait();
    if (on) b3_store_row_chunk(dst, r, mul, FMT);
  } else {
    uint32_t r[16];
    tmem_ld_32x16(taddr, r);
    tmem_ld_wait();
    if (on) b3_store_row_chunk(dst, r, mul, FMT);
  }
}

// ----------------------------------------------------------------------------------------
// dV[kv tile, kv head] = sum P^T dO ,  dK = scale * sum dS^T Q
// ----------------------------------------------------------------------------------------
template <int D, int FMT>
__global__ void __launch_bounds__(B3_THREADS, 1)
attn_bwd_dkv3_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                     const AttnBwd3Params p) {
  using Cfg = AttnBwd3Cfg<D>;
  constexpr int NH = D / 64;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sK = base;
  const uint32_t sV = base + Cfg::kTileBytes;
  auto sQ = [&](int s) { return base + Cfg::kTileBytes * (2 + 2 * s); };
  auto sdO = [&](int s) { return base + Cfg::kTileBytes * (3 + 2 * s); };
  const uint32_t scal = base + Cfg::kTileBytes * 6;
  const uint32_t bars = scal + Cfg::kScalarBytes;
  const uint32_t bar_kv = bars;
  auto bar_qdo_full = [&](int s) { return bars + 8u * (1 + s); };
  auto bar_qdo_empty = [&](int s) { return bars + 8u * (3 + s); };
  const uint32_t bar_s_full = bars + 8u * 5, bar_dp_full = bars + 8u * 6;
  const uint32_t bar_pa_full = bars + 8u * 7, bar_pb_full = bars + 8u * 8;
  const uint32_t bar_acc_done = bars + 8u * 9;
  const uint32_t holder = bars + 8u * 10;
  float* scal_f = reinterpret_cast<float*>(smem_raw + (scal - smem_u32(smem_raw)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kt = blockIdx.x / p.nkv;  // early tiles have the most queries: they start first, heads fastest
  const int hk = blockIdx.x % p.nkv;
  const int G = p.nh / p.nkv;
  const int k0 = kt * B3_T;
  const int k_last = min(k0 + B3_T - 1, p.T - 1);
  const int de_last = p.doc_end[k_last];
  const int qb_lo = kt;
  const int qb_hi = (de_last - 1) / B3_T;
  const int nq = qb_hi - qb_lo + 1;
  const int niter = nq * G;

  if (warp == 1 && lane == 0) {
    mbar_init(bar_kv, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_qdo_full(s), 1);
      mbar_init(bar_qdo_empty(s), 1);
    }
    mbar_init(bar_s_full, 1);
    mbar_init(bar_dp_full, 1);
    mbar_init(bar_pa_full, B3_CW);
    mbar_init(bar_pb_full, B3_CW);
    mbar_init(bar_acc_done, 1);
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
  const uint32_t tS = tmem, tdP = tmem + 128u, tdV = tmem + 256u, tdK = tmem + 256u + D;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar_kv, 2 * Cfg::kTileBytes);
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        tma_load_2d(sK + h * Cfg::kHalfBytes, &tmK, bar_kv, hk * D + 64 * h, k0);
        tma_load_2d(sV + h * Cfg::kHalfBytes, &tmV, bar_kv, hk * D + 64 * h, k0);
      }
      for (int it = 0; it < niter; ++it) {
        const int s = it & 1;
        if (!mbar_wait(bar_qdo_empty(s), ((it >> 1) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        const int head = hk * G + it / nq;
        const int q0 = (qb_lo + it % nq) * B3_T;
        mbar_expect_tx(bar_qdo_full(s), 2 * Cfg::kTileBytes);
#pragma unroll
        for (int h = 0; h < NH; ++h) {
          tma_load_2d(sQ(s) + h * Cfg::kHalfBytes, &tmQ, bar_qdo_full(s), head * D + 64 * h, q0);
          tma_load_2d(sdO(s) + h * Cfg::kHalfBytes, &tmdO, bar_qdo_full(s), head * D + 64 * h, q0);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc_s = make_idesc_f16(128, 128, FMT, 0, 0);
      const uint32_t idesc_g = make_idesc_f16(128, D, FMT, 0, 1);
      const SmemDescBase dK = make_smem_desc_base(sK, 16, 1024), dV = make_smem_desc_base(sV, 16, 1024);
      auto issue_s = [&](int s) {  // S^T = K Q^T
        const SmemDescBase dQ = make_smem_desc_base(sQ(s), 16, 1024);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = (ks / 4) * Cfg::kHalfBytes + (ks % 4) * 32;
          tc_mma_f16(tS, smem_desc_at(dK, off), smem_desc_at(dQ, off), idesc_s, ks != 0);
        }
        tc_commit(bar_s_full);
      };
      auto issue_dp = [&](int s) {  // dP^T = V dO^T
        const SmemDescBase ddO = make_smem_desc_base(sdO(s), 16, 1024);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = (ks / 4) * Cfg::kHalfBytes + (ks % 4) * 32;
          tc_mma_f16(tdP, smem_desc_at(dV, off), smem_desc_at(ddO, off), idesc_s, ks != 0);
        }
        tc_commit(bar_dp_full);
      };
      auto issue_acc = [&](uint32_t acc, uint32_t a_tmem, uint32_t b_tile, bool first) {  // acc += A[tmem] . B[tile]
        const SmemDescBase b = make_smem_desc_base(b_tile, Cfg::kHalfBytes, 1024);
        tc_mma_f16_ts(acc, a_tmem + b3_pcol(0), smem_desc_at(b, 0), idesc_g, first ? 0u : 1u);
#pragma unroll
        for (int ks = 1; ks < 8; ++ks) tc_mma_f16_ts(acc, a_tmem + b3_pcol(ks), smem_desc_at(b, ks * 2048), idesc_g, 1u);
      };
      bool ok = mbar_wait(bar_kv, 0, p.status, kTimeoutMma);
      if (ok) ok = mbar_wait(bar_qdo_full(0), 0, p.status, kTimeoutMma);
      if (ok) {
        tc_fence_after();
        issue_s(0);
        issue_dp(0);
      }
      for (int it = 0; it < niter && ok; ++it) {
        const int s = it & 1;
        const bool more = it + 1 < niter;
        if (!mbar_wait(bar_pa_full, it & 1, p.status, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        issue_acc(tdV, tS, sdO(s), it == 0);
        if (more) {
          if (!mbar_wait(bar_qdo_full(s ^ 1), ((it + 1) >> 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          issue_s(s ^ 1);
        }
        if (!mbar_wait(bar_pb_full, it & 1, p.status, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        issue_acc(tdK, tdP, sQ(s), it == 0);
        tc_commit(bar_qdo_empty(s));
        if (more) issue_dp(s ^ 1);
      }
      if (ok) tc_commit(bar_acc_done);
    }
  } else {
    const int quarter = warp & 3;
    const int cq = (warp - 2) >> 2;  // columns [32 cq, 32 cq + 32)
    const int ctid = threadIdx.x - 64;
    const int kr = k0 + quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const float LOG2E = 1.4426950408889634f;
    const float sl2 = p.scale * LOG2E;
    const uint64_t sl2x2 = pack_f32x2(sl2, sl2);
    auto fetch = [&](int it, float& f, int& i) {
      const int head = hk * G + it / nq;
      const int t = (qb_lo + it % nq) * B3_T + (ctid & 127);
      if (ctid < 128) {
        f = t < p.T ? p.lse[(long long)head * p.T + t] * LOG2E : 0.f;
        i = t < p.T ? p.doc_start[t] : 0x7fffffff;
      } else if (ctid < 256) {
        f = t < p.T ? p.delta[(long long)head * p.T + t] : 0.f;
        i = 0;
      }
    };
    auto publish = [&](int buf, float f, int i) {
      float* b = scal_f + buf * 384;
      if (ctid < 256) b[ctid] = -f;  // [0,128): -lse*log2e, [128,256): -delta
      if (ctid < 128) reinterpret_cast<int*>(b)[256 + ctid] = i;
    };
    float nf = 0.f;
    int ni = 0;
    fetch(0, nf, ni);
    publish(0, nf, ni);
    b3_compute_sync();
    bool ok = true;
    const int c0 = cq * 32;
    for (int it = 0; it < niter; ++it) {
      const bool more = it + 1 < niter;
      if (more) fetch(it + 1, nf, ni);
      const float* b = scal_f + (it & 1) * 384;
      const int* bi = reinterpret_cast<const int*>(b) + 256;
      const int q0 = (qb_lo + it % nq) * B3_T;
      const bool need_mask = !(q0 >= k0 + B3_T - 1 && bi[127] <= k0);
      uint32_t pk[16];
      // ---- stage A: P^T from S^T
      if (ok && !mbar_wait(bar_s_full, it & 1, p.status, kTimeoutEpilogue)) ok = false;
      if (ok) {
        tc_fence_after();
        {
          uint32_t rs[32];
          tmem_ld_32x32(tS + lane_addr + c0, rs);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const int col = c0 + i;
            const float4 l4 = *reinterpret_cast<const float4*>(b + col);
            float pv[4];
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), sl2x2, pack_f32x2(l4.x, l4.y)), pv[0], pv[1]);
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[i + 2]), __uint_as_float(rs[i + 3])), sl2x2, pack_f32x2(l4.z, l4.w)), pv[2], pv[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) pv[e] = fast_exp2(pv[e]);
            if (need_mask) {
              const int4 s4 = *reinterpret_cast<const int4*>(bi + col);
              const int t = q0 + col;
              if (!(kr >= s4.x && kr <= t)) pv[0] = 0.f;
              if (!(kr >= s4.y && kr <= t + 1)) pv[1] = 0.f;
              if (!(kr >= s4.z && kr <= t + 2)) pv[2] = 0.f;
              if (!(kr >= s4.w && kr <= t + 3)) pv[3] = 0.f;
            }
            pk[i / 2] = b3_pack2(pv[0], pv[1], FMT);
            pk[i / 2 + 1] = b3_pack2(pv[2], pv[3], FMT);
          }
        }
        tmem_st_32x16(tS + lane_addr + c0, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_pa_full);
      }
      // ---- stage B: dS^T = P^T o (dP^T - delta)
      if (ok && !mbar_wait(bar_dp_full, it & 1, p.status, kTimeoutEpilogue)) ok = false;
      if (ok) {
        tc_fence_after();
        uint32_t dk[16];
        {
          uint32_t rp[32];
          tmem_ld_32x32(tdP + lane_addr + c0, rp);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(b + 128 + c0 + i);
            float p0, p1, p2, p3;
            b3_unpack2(pk[i / 2], FMT, p0, p1);
            b3_unpack2(pk[i / 2 + 1], FMT, p2, p3);
            unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), add_f32x2(pack_f32x2(__uint_as_float(rp[i]), __uint_as_float(rp[i + 1])), pack_f32x2(d4.x, d4.y))), p0, p1);
            unpack_f32x2(mul_f32x2(pack_f32x2(p2, p3), add_f32x2(pack_f32x2(__uint_as_float(rp[i + 2]), __uint_as_float(rp[i + 3])), pack_f32x2(d4.z, d4.w))), p2, p3);
            dk[i / 2] = b3_pack2(p0, p1, FMT);
            dk[i / 2 + 1] = b3_pack2(p2, p3, FMT);
          }
        }
        tmem_st_32x16(tdP + lane_addr + c0, dk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_pb_full);
      }
      if (more) publish((it + 1) & 1, nf, ni);
      b3_compute_sync();
    }
    if (ok && mbar_wait(bar_acc_done, 0, p.status, kTimeoutEpilogue)) {
      tc_fence_after();
      const int col = cq * (D / 4);
      const bool on = kr < p.T;
      b3_store_quarter<D, FMT>(reinterpret_cast<uint16_t*>(p.dv) + (long long)kr * p.lddv + hk * D + col, tdV + lane_addr + col,
                               1.f, on);
      b3_store_quarter<D, FMT>(reinterpret_cast<uint16_t*>(p.dk) + (long long)kr * p.lddk + hk * D + col, tdK + lane_addr + col,
                               p.scale, on);
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
// dQ[q tile, head] = scale * sum_j dS_j K_j
// ----------------------------------------------------------------------------------------
template <int D, int FMT>
__global__ void __launch_bounds__(B3_THREADS, 1)
attn_bwd_dq3_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const AttnBwd3Params p) {
  using Cfg = AttnBwd3Cfg<D>;
  constexpr int NH = D / 64;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = base;
  const uint32_t sdO = base + Cfg::kTileBytes;
  auto sK = [&](int s) { return base + Cfg::kTileBytes * (2 + 2 * s); };
  auto sV = [&](int s) { return base + Cfg::kTileBytes * (3 + 2 * s); };
  const uint32_t bars = base + Cfg::kTileBytes * 6 + Cfg::kScalarBytes;
  const uint32_t bar_q = bars;
  auto bar_k_full = [&](int s) { return bars + 8u * (1 + s); };
  auto bar_k_empty = [&](int s) { return bars + 8u * (3 + s); };
  auto bar_v_full = [&](int s) { return bars + 8u * (5 + s); };
  auto bar_v_empty = [&](int s) { return bars + 8u * (7 + s); };
  const uint32_t bar_s_full = bars + 8u * 9, bar_sa_done = bars + 8u * 10, bar_acc_done = bars + 8u * 11;
  auto bar_dp_full = [&](int b) { return bars + 8u * (12 + b); };
  auto bar_pb_full = [&](int b) { return bars + 8u * (14 + b); };
  const uint32_t holder = bars + 8u * 16;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = gridDim.x / p.nh - 1 - blockIdx.x / p.nh;  // long tiles (late in their document) first, heads fastest
  const int head = blockIdx.x % p.nh;
  const int hk = head / (p.nh / p.nkv);
  const int q0 = qt * B3_T;
  const int q_last = min(q0 + B3_T - 1, p.T - 1);
  const int ds_last = p.doc_start[q_last];
  const int kb_lo = p.doc_start[q0] / B3_T;
  const int nblk = q_last / B3_T - kb_lo + 1;

  if (warp == 1 && lane == 0) {
    mbar_init(bar_q, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_k_full(s), 1);
      mbar_init(bar_k_empty(s), 1);
      mbar_init(bar_v_full(s), 1);
      mbar_init(bar_v_empty(s), 1);
      mbar_init(bar_dp_full(s), 1);
      mbar_init(bar_pb_full(s), B3_CW);
    }
    mbar_init(bar_s_full, 1);
    mbar_init(bar_sa_done, B3_CW);
    mbar_init(bar_acc_done, 1);
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
  const uint32_t tS = tmem, tdQ = tmem + 384u;
  auto tdP = [&](int b) { return tmem + 128u + 128u * b; };

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar_q, 2 * Cfg::kTileBytes);
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        tma_load_2d(sQ + h * Cfg::kHalfBytes, &tmQ, bar_q, head * D + 64 * h, q0);
        tma_load_2d(sdO + h * Cfg::kHalfBytes, &tmdO, bar_q, head * D + 64 * h, q0);
      }
      for (int j = 0; j < nblk; ++j) {
        const int s = j & 1;
        const uint32_t par = ((j >> 1) & 1) ^ 1u;
        const int k0 = (kb_lo + j) * B3_T;
        if (!mbar_wait(bar_v_empty(s), par, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(bar_v_full(s), Cfg::kTileBytes);
#pragma unroll
        for (int h = 0; h < NH; ++h) tma_load_2d(sV(s) + h * Cfg::kHalfBytes, &tmV, bar_v_full(s), hk * D + 64 * h, k0);
        if (!mbar_wait(bar_k_empty(s), par, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(bar_k_full(s), Cfg::kTileBytes);
#pragma unroll
        for (int h = 0; h < NH; ++h) tma_load_2d(sK(s) + h * Cfg::kHalfBytes, &tmK, bar_k_full(s), hk * D + 64 * h, k0);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc_s = make_idesc_f16(128, 128, FMT, 0, 0);
      const uint32_t idesc_g = make_idesc_f16(128, D, FMT, 0, 1);
      auto issue_scores = [&](uint32_t acc, uint32_t a_tile, uint32_t b_tile, uint32_t bar) {  // acc = A . B^T
        const SmemDescBase a = make_smem_desc_base(a_tile, 16, 1024), b = make_smem_desc_base(b_tile, 16, 1024);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = (ks / 4) * Cfg::kHalfBytes + (ks % 4) * 32;
          tc_mma_f16(acc, smem_desc_at(a, off), smem_desc_at(b, off), idesc_s, ks != 0 ? 1u : 0u);
        }
        tc_commit(bar);
      };
      auto issue_dq = [&](int s, bool first) {  // dQ += dS K
        const SmemDescBase b = make_smem_desc_base(sK(s), Cfg::kHalfBytes, 1024);
        const uint32_t ds = tdP(s);
        tc_mma_f16_ts(tdQ, ds + b3_pcol(0), smem_desc_at(b, 0), idesc_g, first ? 0u : 1u);
#pragma unroll
        for (int ks = 1; ks < 8; ++ks) tc_mma_f16_ts(tdQ, ds + b3_pcol(ks), smem_desc_at(b, ks * 2048), idesc_g, 1u);
      };
      const bool tr = blockIdx.x == gridDim.x / p.nh / 2 * p.nh;
      FMSB_TRACE3(tr, 4000);
      bool ok = mbar_wait(bar_q, 0, p.status, kTimeoutMma);
      FMSB_TRACE3(tr, 4001);
      for (int j = -1; j < nblk && ok; ++j) {
        FMSB_TRACE3(tr, 4096 + 8 * (j + 1) + 0);
        if (j + 1 < nblk) {
          const int n = j + 1, s = n & 1;
          const uint32_t par = (n >> 1) & 1;
          // S(j) is in the compute warps' registers: S(j+1) may overwrite it while they work
          if (j >= 0 && !mbar_wait(bar_sa_done, j & 1, p.status, kTimeoutMma)) { ok = false; break; }
          if (!mbar_wait(bar_k_full(s), par, p.status, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          FMSB_TRACE3(tr, 4096 + 8 * (j + 1) + 1);
          issue_scores(tS, sQ, sK(s), bar_s_full);
          if (!mbar_wait(bar_v_full(s), par, p.status, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          // dS(j-1) in this buffer has been read: dQ(j-1) was issued before this product
          issue_scores(tdP(s), sdO, sV(s), bar_dp_full(s));
          tc_commit(bar_v_empty(s));
          FMSB_TRACE3(tr, 4096 + 8 * (j + 1) + 2);
        }
        if (j >= 0) {
          const int s = j & 1;
          if (!mbar_wait(bar_pb_full(s), (j >> 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          FMSB_TRACE3(tr, 4096 + 8 * (j + 1) + 3);
          issue_dq(s, j == 0);
          tc_commit(bar_k_empty(s));
          FMSB_TRACE3(tr, 4096 + 8 * (j + 1) + 4);
        }
      }
      if (ok) tc_commit(bar_acc_done);
      FMSB_TRACE3(tr, 4003);
    }
  } else {
    const int quarter = warp & 3;
    const int cq = (warp - 2) >> 2;  // columns [32 cq, 32 cq + 32)
    const int row = quarter * 32 + lane;
    const int t = q0 + row;
    const bool row_ok = t < p.T;
    const int ds = row_ok ? p.doc_start[t] : 0;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const float LOG2E = 1.4426950408889634f;
    const float sl2 = p.scale * LOG2E;
    const float lse2 = row_ok ? p.lse[(long long)head * p.T + t] * LOG2E : 0.f;
    const float dlt = row_ok ? p.delta[(long long)head * p.T + t] : 0.f;
    const uint64_t sl2x2 = pack_f32x2(sl2, sl2), nlse2 = pack_f32x2(-lse2, -lse2), ndlt2 = pack_f32x2(-dlt, -dlt);
    const int c0 = cq * 32;
    const bool trc = blockIdx.x == gridDim.x / p.nh / 2 * p.nh && threadIdx.x == 64;
    bool ok = true;
    FMSB_TRACE3(trc, 12);
    for (int j = 0; j < nblk && ok; ++j) {
      const int k0 = (kb_lo + j) * B3_T;
      const bool need_mask = !(q0 >= k0 + B3_T - 1 && ds_last <= k0) || !row_ok;
      FMSB_TRACE3(trc, 64 + 8 * j + 0);
      if (!mbar_wait(bar_s_full, j & 1, p.status, kTimeoutEpilogue)) { ok = false; break; }
      tc_fence_after();
      FMSB_TRACE3(trc, 64 + 8 * j + 1);
      uint32_t pk[16];
      {
        uint32_t rs[32];
        tmem_ld_32x32(tS + lane_addr + c0, rs);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_sa_done);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p0, p1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), sl2x2, nlse2), p0, p1);
          p0 = fast_exp2(p0);
          p1 = fast_exp2(p1);
          if (need_mask) {
            const int kk = k0 + c0 + i;
            if (!(row_ok && kk >= ds && kk <= t)) p0 = 0.f;
            if (!(row_ok && kk + 1 >= ds && kk + 1 <= t)) p1 = 0.f;
          }
          pk[i / 2] = b3_pack2(p0, p1, FMT);
        }
      }
      FMSB_TRACE3(trc, 64 + 8 * j + 2);
      if (!mbar_wait(bar_dp_full(j & 1), (j >> 1) & 1, p.status, kTimeoutEpilogue)) { ok = false; break; }
      tc_fence_after();
      FMSB_TRACE3(trc, 64 + 8 * j + 3);
      uint32_t dk[16];
      const uint32_t tdp = tdP(j & 1) + lane_addr + c0;
      {
        uint32_t rp[32];
        tmem_ld_32x32(tdp, rp);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p0, p1;
          b3_unpack2(pk[i / 2], FMT, p0, p1);
          unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), add_f32x2(pack_f32x2(__uint_as_float(rp[i]), __uint_as_float(rp[i + 1])), ndlt2)), p0, p1);
          dk[i / 2] = b3_pack2(p0, p1, FMT);
        }
      }
      tmem_st_32x16(tdp, dk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_pb_full(j & 1));
      FMSB_TRACE3(trc, 64 + 8 * j + 4);
    }
    FMSB_TRACE3(trc, 13);
    if (ok && mbar_wait(bar_acc_done, 0, p.status, kTimeoutEpilogue)) {
      tc_fence_after();
      FMSB_TRACE3(trc, 14);
      const int col = cq * (D / 4);
      b3_store_quarter<D, FMT>(reinterpret_cast<uint16_t*>(p.dq) + (long long)t * p.lddq + head * D + col,
                               tdQ + lane_addr + col, p.scale, row_ok);
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

}  // namespace fmsb

using namespace fmsb;

#ifdef FMSB_TRACE
extern "C" int fmsb_attn_trace3_read(long long* host, int n) {
  if (n > 8192) n = 8192;
  return (int)cudaMemcpyFromSymbol(host, fmsb::g_trace3, sizeof(long long) * n);
}
#endif

static int b3_make_maps(CUtensorMap* tq, CUtensorMap* tk, CUtensorMap* tv, CUtensorMap* tdo, const void* q,
                        long long ldq, const void* k, long long ldk, const void* v, long long ldv, const void* dout,
                        long long lddo, int T, int nh, int nkv, int d) {
  using namespace fmsb_host;
  int rc;
  if ((rc = make_tmap_2d_16b(tq, q, T, (uint64_t)nh * d, ldq, 128, 64))) return rc;
  if ((rc = make_tmap_2d_16b(tk, k, T, (uint64_t)nkv * d, ldk, 128, 64))) return rc;
  if ((rc = make_tmap_2d_16b(tv, v, T, (uint64_t)nkv * d, ldv, 128, 64))) return rc;
  if ((rc = make_tmap_2d_16b(tdo, dout, T, (uint64_t)nh * d, lddo, 128, 64))) return rc;
  return 0;
}

template <typename K>
static int b3_set_smem(K kern, int bytes) {
  return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

extern "C" int fmsb_attn_bwd_dq3(const void* q, long long ldq, const void* k, long long ldk, const void* v,
                                 long long ldv, const void* dout, long long lddo, void* dq, long long lddq,
                                 const float* lse, const float* delta, const int* doc_start, const int* doc_end,
                                 int T, int nh, int nkv, int d, float scale, int fmt, int* status,
                                 cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!(d == 64 || d == 128) || nh % nkv != 0) return -2;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || (lddq % 8)) return -2;
  CUtensorMap tq, tk, tv, tdo;
  int rc = b3_make_maps(&tq, &tk, &tv, &tdo, q, ldq, k, ldk, v, ldv, dout, lddo, T, nh, nkv, d);
  if (rc) return rc;
  AttnBwd3Params p{};
  p.T = T; p.nh = nh; p.nkv = nkv; p.d = d; p.scale = scale;
  p.doc_start = doc_start; p.doc_end = doc_end; p.lse = lse; p.delta = delta;
  p.dq = dq; p.lddq = lddq; p.fmt = fmt; p.status = status;
  const long long ctas = (long long)nh * ((T + B3_T - 1) / B3_T);
  if (ctas > 0x7fffffffLL) return -2;
  const dim3 grid((unsigned)ctas);
#define FMSB_B3(DD, FF)                                                                                          \
  do {                                                                                                           \
    static bool cfg = false;                                                                                     \
    if (!cfg) {                                                                                                  \
      if ((rc = b3_set_smem(attn_bwd_dq3_kernel<DD, FF>, AttnBwd3Cfg<DD>::kSmemBytes))) return rc;             \
      cfg = true;                                                                                                \
    }                                                                                                            \
    attn_bwd_dq3_kernel<DD, FF><<<grid, B3_THREADS, AttnBwd3Cfg<DD>::kSmemBytes, stream>>>(tq, tk, tv, tdo, p);       \
  } while (0)
  if (d == 128 && fmt == 1) FMSB_B3(128, 1);
  else if (d == 128) FMSB_B3(128, 0);
  else if (fmt == 1) FMSB_B3(64, 1);
  else FMSB_B3(64, 0);
#undef FMSB_B3
  return (int)cudaGetLastError();
}

extern "C" int fmsb_attn_bwd_dkv3(const void* q, long long ldq, const void* k, long long ldk, const void* v,
                                  long long ldv, const void* dout, long long lddo, void* dk, long long lddk, void* dv,
                                  long long lddv, const float* lse, const float* delta, const int* doc_start,
                                  const int* doc_end, int T, int nh, int nkv, int d, float scale, int fmt,
                                  int* status, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!(d == 64 || d == 128) || nh % nkv != 0) return -2;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || (lddk % 8) || (lddv % 8)) return -2;
  CUtensorMap tq, tk, tv, tdo;
  int rc = b3_make_maps(&tq, &tk, &tv, &tdo, q, ldq, k, ldk, v, ldv, dout, lddo, T, nh, nkv, d);
  if (rc) return rc;
  AttnBwd3Params p{};
  p.T = T; p.nh = nh; p.nkv = nkv; p.d = d; p.scale = scale;
  p.doc_start = doc_start; p.doc_end = doc_end; p.lse = lse; p.delta = delta;
  p.dk = dk; p.lddk = lddk; p.dv = dv; p.lddv = lddv; p.fmt = fmt; p.status = status;
  const long long ctas = (long long)nkv * ((T + B3_T - 1) / B3_T);
  if (ctas > 0x7fffffffLL) return -2;
  const dim3 grid((unsigned)ctas);
#define FMSB_B3(DD, FF)                                                                                          \
  do {                                                                                                           \
    static bool cfg = false;                                                                                     \
    if (!cfg) {                                                                                                  \
      if ((rc = b3_set_smem(attn_bwd_dkv3_kernel<DD, FF>, AttnBwd3Cfg<DD>::kSmemBytes))) return rc;             \
      cfg = true;                                                                                                \
    }                                                                                                            \
    attn_bwd_dkv3_kernel<DD, FF><<<grid, B3_THREADS, AttnBwd3Cfg<DD>::kSmemBytes, stream>>>(tq, tk, tv, tdo, p);       \
  } while (0)
  if (d == 128 && fmt == 1) FMSB_B3(128, 1);
  else if (d == 128) FMSB_B3(128, 0);
  else if (fmt == 1) FMSB_B3(64, 1);
  else FMSB_B3(64, 0);
#undef FMSB_B3
  return (int)cudaGetLastError();
}

extern "C" int fmsb_attn_delta(const void* o, const void* dout, long long ldo, long long lddo, float* delta, int T, int nh, int d,
                               int fmt, cudaStream_t stream);

// The whole backward (delta, dQ, dK/dV) in one call: three launches from Python cost the host more than the kernels take at
// 1500 tokens.  delta: scratch of nh * T floats.
extern "C" int fmsb_attn_bwd(const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv,
                             const void* o, long long ldo, const void* dout, long long lddo, void* dq, long long lddq,
                             void* dk, long long lddk, void* dv, long long lddv, const float* lse, float* delta,
                             const int* doc_start, const int* doc_end, int T, int nh, int nkv, int d, float scale, int fmt,
                             int* status, cudaStream_t stream) {
  int rc;
  if ((rc = fmsb_attn_delta(o, dout, ldo, lddo, delta, T, nh, d, fmt, stream))) return rc;
  if ((rc = fmsb_attn_bwd_dq3(q, ldq, k, ldk, v, ldv, dout, lddo, dq, lddq, lse, delta, doc_start, doc_end, T, nh, nkv, d, scale,
                              fmt, status, stream))) return rc;
  return fmsb_attn_bwd_dkv3(q, ldq, k, ldk, v, ldv, dout, lddo, dk, lddk, dv, lddv, lse, delta, doc_start, doc_end, T, nh, nkv,
                            d, scale, fmt, status, stream);
}
