// Fused gather + NF4/FP4 dequantise + GEMM + LoRA for sm_100a:
//
//     y[M, N] = alpha * ( x[M, K] . dequant(Wq)[N, K]^T  +  xa[M, R] . Bl[N, R]^T )
//
// The 4-bit weight never exists in 16 bits in global memory: dequant warps read the packed bytes (two
// values per byte, blocks of 64 values sharing one scale, the scales themselves optionally 8-bit "double
// quantised") straight from where they are stored - this GPU's memory or a PEER's shard of the flat
// packed array, through plain loads over NVLink - expand them with the 16-entry code book and write
// 16-bit values directly into the 128-byte-swizzled shared-memory operand tile that tcgen05.mma reads
// (generic-proxy stores, then fence.proxy.async, then an mbarrier arrive).  The activation tiles come
// in by TMA; the LoRA update (xa = x A^T computed beforehand, Bl = s*B) is accumulated by extra K blocks
// into the same tensor-memory accumulator.
//
// This is the kernel for FEW ROWS (M up to a few hundred: one or two 128-row tiles), where every weight
// byte is used once and the job is to stream 4-bit data at memory / link speed.  With thousands of rows
// each weight tile would be expanded again by every row tile; there the framework dequantises once into
// an L2-resident 16-bit buffer and runs gemm_tcgen05.cu.
//
// The same kernel serves GPTQ int4 weights (template parameter GPTQ): qweight [K/8, N] int32 holds eight consecutive
// k of one output column per word, which is exactly one 16-byte chunk of the K-major operand row; scales [K/g, N]
// and packed zero points [K/g, N/8] are per group of g input features (g a multiple of 64, groups in order).
// A dequant warp reads 32 neighbouring columns per load (coalesced) and writes 32 swizzled rows.  Reference
// counterpart: the fused dequantise-and-matmul Triton kernels of
// fms_acceleration_peft/gptqmodel/nn_modules/triton_utils/kernels.py:105-201.
//
// Reference counterparts (NF4 / FP4): bitsandbytes' cgemm_4bit_inference_naive / dequantize + matmul as called from
// fms_acceleration_foak/fused_ops/unsloth_lora/utils.py:119-136,190-203,262-279 and the NCCL all-gather
// of the FSDP-sharded packed parameter that precedes them.
//
// Roles (320 threads): warp 0 TMA producer (x, and xa/Bl for the LoRA blocks), warp 1 MMA issuer,
// warps 2-9 dequantise W tiles and afterwards run the epilogue.  6- or 8-stage ring.  Every wait is bounded.
//
// This first kernel serves peers' shards, a LoRA pair, fp32 block scales and GPTQ weights (77 x 14336 x 4096, one shard: 95.8 ->
// 66.6 us without the per-block 64-bit divisions and with the tile width chosen by turns of the machine).  A plain local
// weight goes to gemm_q4_tma_kernel (double-quantised) or, up to four rows, to q4_rows_kernel.
#include "common.cuh"

namespace fmsb {

constexpr int Q4_BM = 128;
constexpr int Q4_BK = 64;
constexpr int Q4_MAX_RANKS = 16;
constexpr int Q4_DQ_THREADS = 256;  // 8 dequant warps: two per scheduler, so table look-ups of one hide behind the other

struct Q4Params {
  int M, N, K;
  int kblocks1, kblocks2;
  const uint8_t* shard[Q4_MAX_RANKS];  // flat packed array [N*K/2] split into `world` equal shards
  long long shard_bytes;
  int world;
  const float* absmax;       // [N*K/64] fp32, or null when double quantised
  const uint8_t* absmax_q;   // [N*K/64] codes into code256
  const float* code256;      // [256]
  const float* absmax2;      // [N*K/64/256]
  float offset;
  float code16[16];
  // GPTQ int4 (template parameter GPTQ = 1): W[k, n] = scales[g, n] * (q[k, n] - (zero[g, n] + zero_offset)), g = k / group
  const uint32_t* gq_weight;  // [K/8, N]
  const uint16_t* gq_scales;  // [K/group, N] in the compute format
  const uint32_t* gq_zeros;   // [K/group, N/8]
  int gq_group;               // input features per group: a multiple of 64
  int gq_zero_offset;
  void* D;
  long long ldd;
  float alpha;
  int fmt;  // 0 fp16, 1 bf16
  int* status;
};

template <int BN>
struct Q4Cfg {
  static constexpr int kABytes = Q4_BM * Q4_BK * 2;
  static constexpr int kBBytes = BN * Q4_BK * 2;
  // As many stages as shared memory holds (192 KB of operands): the dequant warps run ahead of the tensor core by a
  // store, a proxy fence and an arrive per K block, and a deeper ring hides the round trip of a stage.
  static constexpr int kStages = BN == 128 ? 6 : 8;
  static constexpr int kSmemBytes = kStages * (kABytes + kBBytes) + 1024 + 512;
};

// Streaming loads of packed weights.  A thread's bytes of one K block are a 16- or 32-byte piece of a row whose
// neighbours along K are needed a few blocks later: ask L2 for the whole 256-byte neighbourhood on a miss so that
// DRAM is read in long bursts and the following K blocks of the row hit in L2.
__device__ __forceinline__ uint4 q4_ld16(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 q4_ld8(const uint8_t* p) {
  uint2 v;
  asm volatile("ld.global.L2::256B.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t q4_ld4(const uint8_t* p) {
  uint32_t v;
  asm volatile("ld.global.L2::256B.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t q4_pack2(float a, float b, int fmt) {
  return fmt == 1 ? pack_bf16x2(a, b) : pack_f16x2(a, b);
}

// 32 accumulator columns of one row to D
__device__ __forceinline__ void q4_store32(const Q4Params& p, int row, int col, const uint32_t (&v)[32]) {
  uint16_t* dst = reinterpret_cast<uint16_t*>(p.D) + (long long)row * p.ldd + col;
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    if (col + i < p.N) {  // N % 8 == 0: a group of 8 columns is in range as a whole
      uint4 u;
      u.x = q4_pack2(__uint_as_float(v[i]) * p.alpha, __uint_as_float(v[i + 1]) * p.alpha, p.fmt);
      u.y = q4_pack2(__uint_as_float(v[i + 2]) * p.alpha, __uint_as_float(v[i + 3]) * p.alpha, p.fmt);
      u.z = q4_pack2(__uint_as_float(v[i + 4]) * p.alpha, __uint_as_float(v[i + 5]) * p.alpha, p.fmt);
      u.w = q4_pack2(__uint_as_float(v[i + 6]) * p.alpha, __uint_as_float(v[i + 7]) * p.alpha, p.fmt);
      *reinterpret_cast<uint4*>(dst + i) = u;
    }
  }
}

template <int BN, int GPTQ>
__global__ void __launch_bounds__(64 + Q4_DQ_THREADS, 1)
gemm_q4_fused_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmXa,
                     const __grid_constant__ CUtensorMap tmBl, const Q4Params p) {
  using Cfg = Q4Cfg<BN>;
  constexpr int Q4_STAGES = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  auto sA = [&](int s) { return base + s * (Cfg::kABytes + Cfg::kBBytes); };
  auto sB = [&](int s) { return base + s * (Cfg::kABytes + Cfg::kBBytes) + Cfg::kABytes; };
  const uint32_t bars = base + Q4_STAGES * (Cfg::kABytes + Cfg::kBBytes);
  auto bar_a_full = [&](int s) { return bars + 8u * s; };
  auto bar_b_full = [&](int s) { return bars + 8u * (Q4_STAGES + s); };
  auto bar_empty = [&](int s) { return bars + 8u * (2 * Q4_STAGES + s); };
  const uint32_t bar_acc = bars + 8u * (3 * Q4_STAGES);
  const uint32_t holder = bar_acc + 8u;
  __shared__ float s_code[16];
  __shared__ float s_code256[256];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * BN;
  const int m0 = blockIdx.y * Q4_BM;
  const int kbt = p.kblocks1 + p.kblocks2;

  if (threadIdx.x < 16) s_code[threadIdx.x] = p.code16[threadIdx.x];
  if (p.absmax_q != nullptr)
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_code256[i] = p.code256[i];
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < Q4_STAGES; ++s) {
      mbar_init(bar_a_full(s), 1);
      mbar_init(bar_b_full(s), Q4_DQ_THREADS / 32);  // one arrival per dequant warp
      mbar_init(bar_empty(s), 1);
    }
    mbar_init(bar_acc, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(holder, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(holder));

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = 0; kb < kbt; ++kb) {
        const int s = kb % Q4_STAGES;
        if (!mbar_wait(bar_empty(s), ((kb / Q4_STAGES) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        if (kb < p.kblocks1) {
          mbar_expect_tx(bar_a_full(s), Cfg::kABytes);
          tma_load_2d(sA(s), &tmX, bar_a_full(s), kb * Q4_BK, m0);
        } else {
          const int k2 = (kb - p.kblocks1) * Q4_BK;
          mbar_expect_tx(bar_a_full(s), Cfg::kABytes + BN * Q4_BK * 2);
          tma_load_2d(sA(s), &tmXa, bar_a_full(s), k2, m0);
          tma_load_2d(sB(s), &tmBl, bar_a_full(s), k2, n0);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_f16(128, BN, p.fmt, 0, 0);
      bool ok = true;
      for (int kb = 0; kb < kbt && ok; ++kb) {
        const int s = kb % Q4_STAGES;
        const uint32_t par = (kb / Q4_STAGES) & 1;
        if (!mbar_wait(bar_a_full(s), par, p.status, kTimeoutMma)) { ok = false; break; }
        if (kb < p.kblocks1 && !mbar_wait(bar_b_full(s), par, p.status, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        const SmemDescBase da = make_smem_desc_base(sA(s), 16, 1024), db = make_smem_desc_base(sB(s), 16, 1024);
#pragma unroll
        for (int ks = 0; ks < Q4_BK / 16; ++ks)
          tc_mma_f16(tmem, smem_desc_at(da, ks * 32), smem_desc_at(db, ks * 32), idesc, (kb | ks) != 0);
        tc_commit(bar_empty(s));
      }
      if (ok) tc_commit(bar_acc);
    }
  } else {
    // ------------------------------------------------------------------ dequantise W tiles [BN rows x 64]
    constexpr int TPR = Q4_DQ_THREADS / BN;  // threads per weight row
    constexpr int EPT = Q4_BK / TPR;     // elements per thread and K block: 32, 16 or 8
    const int tid = threadIdx.x - 64;    // 0..Q4_DQ_THREADS-1
    // NF4 / FP4: a row's bytes are contiguous, neighbouring threads share a row.  GPTQ: a word's neighbours in memory
    // are the same k of the next columns, so neighbouring threads take neighbouring rows of the tile.
    const int r = GPTQ ? tid % BN : tid / TPR;     // row inside the tile
    const int part = GPTQ ? tid / BN : tid % TPR;  // which slice of the row's 64 elements
    const int n = n0 + r;
    const bool row_ok = n < p.N;
    bool ok = true;
    // The packed bytes and the scale code of the next PF K blocks are kept in flight in registers: a weight
    // byte is used exactly once, so the loop is a stream and its speed is set by how many loads are outstanding.
    constexpr int PF = 8;
    constexpr int WPT = EPT / 8;  // 32-bit words (= 16-byte output chunks) per thread and K block
    uint32_t w[PF][WPT];
    uint32_t sq[PF];   // 8-bit code of the block scale (double quantised) or the fp32 scale's bits
    float s2[PF];      // second-level scale of the block
    auto issue = [&](int slot, int kb) {
#pragma unroll
      for (int i = 0; i < WPT; ++i) w[slot][i] = 0u;
      sq[slot] = 0u;
      s2[slot] = 0.f;
      if (!row_ok || kb >= p.kblocks1) return;
      if constexpr (GPTQ) {
        const int g = (kb * Q4_BK) / p.gq_group;
        const uint16_t sc = p.gq_scales[(long long)g * p.N + n];
        sq[slot] = __float_as_uint(p.fmt == 1 ? __uint_as_float((uint32_t)sc << 16) : __half2float(__ushort_as_half(sc)));
        const uint32_t zw = p.gq_zeros[(long long)g * (p.N >> 3) + (n >> 3)];
        s2[slot] = (float)(int)(((zw >> ((n & 7) * 4)) & 15u) + p.gq_zero_offset);
#pragma unroll
        for (int i = 0; i < WPT; ++i)
          w[slot][i] = q4_ld4(reinterpret_cast<const uint8_t*>(p.gq_weight + (long long)(kb * 8 + part * WPT + i) * p.N + n));
        return;
      }
      const long long e0 = (long long)n * p.K + (long long)kb * Q4_BK;  // first element of the 64-block
      const long long blk = e0 >> 6;
      if (p.absmax_q != nullptr) {
        sq[slot] = p.absmax_q[blk];
        s2[slot] = p.absmax2[blk >> 8];
      } else {
        sq[slot] = __float_as_uint(p.absmax[blk]);
      }
      const long long byte_off = (e0 >> 1) + part * (EPT / 2);
      // one shard (the usual case) needs no division: two 64-bit divisions per K block and thread were most of the
      // instructions of this loop
      const uint8_t* src = p.world == 1 ? p.shard[0] + byte_off
                                        : p.shard[byte_off / p.shard_bytes] + (byte_off % p.shard_bytes);
      if constexpr (EPT == 32) {
        const uint4 u0 = q4_ld16(src);
        w[slot][0] = u0.x; w[slot][1] = u0.y; w[slot][2] = u0.z; w[slot][3] = u0.w;
      } else if constexpr (EPT == 16) {
        const uint2 u0 = q4_ld8(src);
        w[slot][0] = u0.x; w[slot][1] = u0.y;
      } else {
        w[slot][0] = q4_ld4(src);
      }
    };
#pragma unroll
    for (int j = 0; j < PF; ++j) issue(j, j);
    for (int kb0 = 0; kb0 < p.kblocks1 && ok; kb0 += PF) {
#pragma unroll
      for (int j = 0; j < PF; ++j) {
        const int kb = kb0 + j;
        if (kb >= p.kblocks1 || !ok) break;
        const int s = kb % Q4_STAGES;
        const float scale = GPTQ ? __uint_as_float(sq[j])
                                 : (p.absmax_q != nullptr ? s_code256[sq[j]] * s2[j] + p.offset : __uint_as_float(sq[j]));
        const float zs = GPTQ ? -s2[j] * scale : 0.f;  // (q - z) * s = q * s - z * s
        if (!mbar_wait(bar_empty(s), ((kb / Q4_STAGES) & 1) ^ 1u, p.status, kTimeoutDequant)) { ok = false; break; }
        // one 32-bit word = 8 values = one 16-byte chunk of the swizzled row
#pragma unroll
        for (int i = 0; i < WPT; ++i) {
          uint32_t o[4];
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const uint32_t byte = (w[j][i] >> (8 * b)) & 0xffu;
            if constexpr (GPTQ)  // low nibble first: the smaller k
              o[b] = q4_pack2(fmaf((float)(byte & 15u), scale, zs), fmaf((float)(byte >> 4), scale, zs), p.fmt);
            else
              o[b] = q4_pack2(s_code[byte >> 4] * scale, s_code[byte & 15] * scale, p.fmt);
          }
          const int chunk = part * WPT + i;  // 0..7 within the row
          const uint32_t addr = sB(s) + static_cast<uint32_t>(r * 128 + ((chunk ^ (r & 7)) << 4));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(o[0]), "r"(o[1]), "r"(o[2]),
                       "r"(o[3])
                       : "memory");
        }
        fence_proxy_async_smem();  // every writer orders its own stores before the tensor core's reads
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_b_full(s));
        issue(j, kb + PF);
      }
    }
    // ------------------------------------------------------------------ epilogue
    if (ok && mbar_wait(bar_acc, 0, p.status, kTimeoutEpilogue)) {
      tc_fence_after();
      const int q = warp & 3;
      const int row = m0 + q * 32 + lane;
      const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
      // two warps share a lane quarter: warps 2-5 take the even 32-column groups, warps 6-9 the odd ones
#pragma unroll 1
      for (int c = (warp - 2) >> 2; c < BN / 32; c += 2) {
        uint32_t v[32];
        tmem_ld_32x32(tmem + lane_addr + c * 32, v);
        tmem_ld_wait();
        if (row < p.M) q4_store32(p, row, n0 + c * 32, v);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}

// ----------------------------------------------------------------------------------------
// The same product for one local, double-quantised NF4 / FP4 weight without a LoRA pair (a plain 4-bit layer), laid out
// for latency.  In the kernel above all eight dequant warps work on one K block at a time, so a block costs one warp's
// whole chain (load, look-up, convert, store, fence, arrive: about 2000 cycles whatever the tile).  Here four groups of
// four warps take K blocks in turn, a thread expands a longer piece of a row (64 values at 128 wide) and nothing is
// outstanding when it fences: the packed bytes come in by TMA (a W stage is [BN rows x 128 bytes] = four K blocks,
// 128-byte swizzle) and the 8-bit scale codes of the tile (BN * K / 64 bytes) are copied to shared memory once.
// 77 x 14336 x 4096: 66.6 -> 36.9 us back to back (43.0 with L2 flushed), 77 x 4096 x 4096 (32 wide): 30.8 -> 22.7 us (26.6);
// what is left at 128 wide is shared memory (look-ups, operand writes and the tensor core's reads: about 850 of 1000 cycles
// per K block).
// ----------------------------------------------------------------------------------------
constexpr int Q4T_GROUPS = 4;           // dequant groups of four warps
constexpr int Q4T_DQ_THREADS = Q4T_GROUPS * 128;

template <int BN>
struct Q4tCfg {
  static constexpr int kABytes = Q4_BM * Q4_BK * 2;
  static constexpr int kBBytes = 2 * BN * Q4_BK * 2;  // two K blocks
  // separate rings: a group may expand its next K block while the tensor core still has to read its last one
  static constexpr int kAStages = 4;
  static constexpr int kBStages = BN == 128 ? 2 : 4;
  static constexpr int kWBytes = BN * 128;
  static constexpr int kWStages = BN == 128 ? 2 : 3;
  static constexpr int kFixed = kAStages * kABytes + kBStages * kBBytes + kWStages * kWBytes + 1024 + 512;
  static constexpr int kStatic = 256 * 16 * 8 + 2048;  // the pair table and the small ones
  static constexpr int kScaleBytes = 227 * 1024 - kStatic - kFixed;  // room for the codes and the second-level scales
};

template <int BN, int FMT>
__global__ void __launch_bounds__(96 + Q4T_DQ_THREADS, 1)
gemm_q4_tma_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Q4Params p) {
  using Cfg = Q4tCfg<BN>;
  constexpr int AS = Cfg::kAStages, BS = Cfg::kBStages, WS = Cfg::kWStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  auto sA = [&](int s) { return base + s * Cfg::kABytes; };
  auto sB = [&](int s) { return base + AS * Cfg::kABytes + s * Cfg::kBBytes; };
  auto sW = [&](int s) { return base + AS * Cfg::kABytes + BS * Cfg::kBBytes + s * Cfg::kWBytes; };
  const uint32_t bars = sW(WS);
  auto bar_a_full = [&](int s) { return bars + 8u * s; };
  auto bar_a_empty = [&](int s) { return bars + 8u * (AS + s); };
  auto bar_b_full = [&](int s) { return bars + 8u * (2 * AS + s); };
  auto bar_b_empty = [&](int s) { return bars + 8u * (2 * AS + BS + s); };
  auto bar_w_full = [&](int s) { return bars + 8u * (2 * AS + 2 * BS + s); };
  auto bar_w_empty = [&](int s) { return bars + 8u * (2 * AS + 2 * BS + WS + s); };
  const uint32_t bar_acc = bars + 8u * (2 * AS + 2 * BS + 2 * WS);
  const uint32_t holder = bar_acc + 8u;
  uint8_t* codes = smem_raw + (bars - smem_u32(smem_raw)) + 512;  // [BN][K / 64]
  // value pairs of a byte, sixteen copies side by side: lane l reads copy l % 16, so the 8-byte reads of a half warp
  // never meet in a bank.  One look-up gives two values (two 4-byte look-ups cost six instructions more per byte).
  __shared__ float2 s_pair[256 * 16];
  __shared__ float s_code[16];
  __shared__ float s_code256[256];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * BN;
  const int m0 = blockIdx.y * Q4_BM;
  const int kbt = p.kblocks1;
  const int rows = min(BN, p.N - n0);
  float* s_abs2 = reinterpret_cast<float*>(codes + ((BN * kbt + 15) & ~15));
  const long long blk0 = (long long)n0 * kbt;  // first scale block of the tile
  const long long grp0 = blk0 >> 8;

  if (warp == 1 && lane == 0) {
    for (int s = 0; s < AS; ++s) {
      mbar_init(bar_a_full(s), 1);
      mbar_init(bar_a_empty(s), 1);
    }
    for (int s = 0; s < BS; ++s) {
      mbar_init(bar_b_full(s), 8);  // four warps for each of the two K blocks
      mbar_init(bar_b_empty(s), 1);
    }
    for (int s = 0; s < WS; ++s) {
      mbar_init(bar_w_full(s), 1);
      mbar_init(bar_w_empty(s), Q4T_DQ_THREADS / 32);
    }
    mbar_init(bar_acc, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(holder, 128);
    tmem_relinquish();
  }
  if (threadIdx.x < 16) s_code[threadIdx.x] = p.code16[threadIdx.x];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) s_code256[i] = p.code256[i];
  {
    const int nb = rows * kbt;
    const uint8_t* src = p.absmax_q + blk0;
    int i0 = 0;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
      i0 = nb & ~15;
      for (int i = threadIdx.x * 16; i < i0; i += blockDim.x * 16)
        *reinterpret_cast<uint4*>(codes + i) = *reinterpret_cast<const uint4*>(src + i);
    }
    for (int i = i0 + threadIdx.x; i < nb; i += blockDim.x) codes[i] = src[i];
    const int ng = (int)(((blk0 + nb - 1) >> 8) - grp0) + 1;
    for (int i = threadIdx.x; i < ng; i += blockDim.x) s_abs2[i] = p.absmax2[grp0 + i];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) s_pair[i] = make_float2(s_code[i >> 8], s_code[(i >> 4) & 15]);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(holder));

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = 0; kb < kbt; ++kb) {
        const int s = kb % AS;
        if (!mbar_wait(bar_a_empty(s), ((kb / AS) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(bar_a_full(s), Cfg::kABytes);
        tma_load_2d(sA(s), &tmX, bar_a_full(s), kb * Q4_BK, m0);
      }
    }
  } else if (warp == 2) {
    // W has a producer of its own: behind the waits for free activation stages it was asked for too late
    if (lane == 0) {
      for (int wi = 0; 4 * wi < kbt; ++wi) {
        const int s = wi % WS;
        if (!mbar_wait(bar_w_empty(s), ((wi / WS) & 1) ^ 1u, p.status, kTimeoutProducer)) break;
        mbar_expect_tx(bar_w_full(s), Cfg::kWBytes);
        tma_load_2d(sW(s), &tmW, bar_w_full(s), wi * 64, n0);  // 64 16-bit units = 128 bytes = 256 weights
      }
    }
  } else if (warp == 1) {
    // Two K blocks per hand-off: the issuing thread needs about 700 cycles for two waits, four short products and two
    // commits, more than four products of 128 x BN x 16 take.
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc_f16(128, BN, FMT, 0, 0);
    bool ok = true;
    for (int st = 0; 2 * st < kbt && ok; ++st) {
      const int sb = st % BS;
      if (!mbar_wait(bar_b_full(sb), (st / BS) & 1, p.status, kTimeoutMma)) { ok = false; break; }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int kb = 2 * st + j;
        if (kb >= kbt) break;
        const int sa = kb % AS;
        if (!mbar_wait(bar_a_full(sa), (kb / AS) & 1, p.status, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        const SmemDescBase da = make_smem_desc_base(sA(sa), 16, 1024);
        const SmemDescBase db = make_smem_desc_base(sB(sb) + j * (BN * 128), 16, 1024);
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < Q4_BK / 16; ++ks)
            tc_mma_f16(tmem, smem_desc_at(da, ks * 32), smem_desc_at(db, ks * 32), idesc, (kb | ks) != 0);
          tc_commit(bar_a_empty(sa));
        }
      }
      if (ok && leader) tc_commit(bar_b_empty(sb));
    }
    if (ok && leader) tc_commit(bar_acc);
  } else {
    // ------------------------------------------------------------------ dequantise W tiles [BN rows x 64]
    constexpr int TPR = 128 / BN;   // threads per weight row
    constexpr int CPT = 8 / TPR;    // 16-byte output chunks (= 4-byte packed words) per thread and K block
    const int tid = threadIdx.x - 96;
    const int group = tid >> 7;
    const int r = (tid & 127) / TPR, part = (tid & 127) % TPR;
    const uint32_t copy = (lane & 15) * 8;
    const bool row_ok = r < rows;
    const long long rb0 = blk0 + (long long)r * kbt;
    bool ok = true;
    const int kb_end = (kbt + 1) & ~1;  // an odd last block: its partner only arrives
    for (int kb = group; kb < kb_end; kb += Q4T_GROUPS) {  // group g of a W stage takes its K block g
      const int wi = kb >> 2, ws = wi % WS;
      if (!mbar_wait(bar_w_full(ws), (wi / WS) & 1, p.status, kTimeoutDequant)) { ok = false; break; }
      // packed bytes of this thread: 4 * CPT of the row's 32 for this K block, in the swizzled 128-byte row
      const int byte = group * 32 + part * (4 * CPT);
      uint32_t w[CPT];
#pragma unroll
      for (int i = 0; i < CPT; i += 4) {
        const int bi = byte + 4 * i;
        const uint32_t wa = sW(ws) + static_cast<uint32_t>(r * 128 + (((bi >> 4) ^ (r & 7)) << 4) + (bi & 15));
        if constexpr (CPT >= 4)
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[i]), "=r"(w[i + 1]), "=r"(w[i + 2]), "=r"(w[i + 3]) : "r"(wa));
        else
          asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(w[i]), "=r"(w[i + 1]) : "r"(wa));
      }
      float scale = 0.f;
      if (row_ok && kb < kbt) scale = s_code256[codes[r * kbt + kb]] * s_abs2[(int)(((rb0 + kb) >> 8) - grp0)] + p.offset;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_w_empty(ws));
      const int st = kb >> 1, s = st % BS;
      if (!mbar_wait(bar_b_empty(s), ((st / BS) & 1) ^ 1u, p.status, kTimeoutDequant)) { ok = false; break; }
      const uint64_t scale2 = pack_f32x2(scale, scale);
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        uint32_t o[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const uint32_t off = ((b == 0 ? w[i] << 7 : w[i] >> (8 * b - 7)) & 0x7f80u) | copy;
          const float2 v = *reinterpret_cast<const float2*>(reinterpret_cast<const uint8_t*>(s_pair) + off);
          float v0, v1;
          unpack_f32x2(mul_f32x2(pack_f32x2(v.x, v.y), scale2), v0, v1);
          o[b] = q4_pack2(v0, v1, FMT);
        }
        const int chunk = part * CPT + i;
        const uint32_t addr = sB(s) + static_cast<uint32_t>((kb & 1) * (BN * 128) + r * 128 + ((chunk ^ (r & 7)) << 4));
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                     : "memory");
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_b_full(s));
    }
    if (ok && mbar_wait(bar_acc, 0, p.status, kTimeoutEpilogue)) {
      tc_fence_after();
      const int q = warp & 3;
      const int row = m0 + q * 32 + lane;
      const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
#pragma unroll 1
      for (int c = (warp - 3) >> 2; c < BN / 32; c += Q4T_GROUPS) {
        uint32_t v[32];
        tmem_ld_32x32(tmem + lane_addr + c * 32, v);
        tmem_ld_wait();
        if (row < p.M) q4_store32(p, row, n0 + c * 32, v);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}

// ----------------------------------------------------------------------------------------
// A few rows (decoding): y[m, n] = alpha * sum_k x[m, k] w[n, k], M <= 4, on the CUDA cores.
//
// A tensor-core tile computes 128 rows whatever M is, and its operand path (registers, shared memory, proxy fence,
// barrier, MMA) is a chain of 64 hand-offs for K = 4096.  Here a warp streams whole rows of W: a lane takes 16 packed
// bytes (32 values of one scale block), looks the codes up in a 16-word shared table (conflict-free), multiplies
// them with x in fp32 and applies the block's scale once per 32 products.  x lies in shared memory as fp32, ordered so
// that the 16-byte reads of a warp are contiguous.  What bounds it is issue: about four instructions per weight
// (two to extract, one look-up, one fused multiply-add).  1 x 4096 x 4096, NF4: 7.9 us back to back (about 12.5
// with L2 flushed) against 44.5 us for the tensor-core form it replaces there.
// ----------------------------------------------------------------------------------------
constexpr int Q4V_WARPS = 8;

template <int M, int ROWS, int FMT>
__global__ void __launch_bounds__(Q4V_WARPS * 32)
q4_rows_kernel(const uint16_t* __restrict__ x, long long ldx, const Q4Params p) {
  extern __shared__ float4 xs[];  // [M][8][K / 32]: the j-th four values of 32-value group i at (m * 8 + j) * groups + i
  __shared__ float s_code[16];
  __shared__ float s_code256[256];
  const int groups = p.K >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * Q4V_WARPS + warp) * ROWS;
  const uint8_t* wp = p.shard[0];
  const bool dq = p.absmax_q != nullptr;
  // the weights of the first step are on their way while x is laid out
  uint4 w[ROWS];
  float sc[ROWS];
  uint32_t sq[ROWS];
  auto issue = [&](int i) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      w[r] = make_uint4(0u, 0u, 0u, 0u);
      sq[r] = 0u;
      sc[r] = 0.f;
      if (i < groups && n0 + r < p.N) {
        const long long g = (long long)(n0 + r) * groups + i;
        w[r] = q4_ld16(wp + g * 16);
        if (dq) {
          sq[r] = p.absmax_q[g >> 1];
          sc[r] = p.absmax2[g >> 9];
        } else {
          sc[r] = p.absmax[g >> 1];
        }
      }
    }
  };
  issue(lane);
  if (threadIdx.x < 16) s_code[threadIdx.x] = p.code16[threadIdx.x];
  if (dq)
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_code256[i] = p.code256[i];
#pragma unroll
  for (int m = 0; m < M; ++m)
    for (int v = threadIdx.x; v < p.K / 8; v += blockDim.x) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + m * ldx + v * 8);
      const uint32_t uw[4] = {u.x, u.y, u.z, u.w};
      float f[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (FMT == 1) {
          f[2 * j] = __uint_as_float(uw[j] << 16);
          f[2 * j + 1] = __uint_as_float(uw[j] & 0xffff0000u);
        } else {
          const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&uw[j]));
          f[2 * j] = h.x;
          f[2 * j + 1] = h.y;
        }
      }
      const int i = v >> 2, j = (v & 3) * 2;
      xs[(m * 8 + j) * groups + i] = make_float4(f[0], f[1], f[2], f[3]);
      xs[(m * 8 + j + 1) * groups + i] = make_float4(f[4], f[5], f[6], f[7]);
    }
  __syncthreads();
  float acc[ROWS][M];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
  for (int i = lane; i < groups; i += 32) {
    uint4 cw[ROWS];
    float scale[ROWS], part[ROWS][M];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      cw[r] = w[r];
      scale[r] = dq ? s_code256[sq[r]] * sc[r] + p.offset : sc[r];
#pragma unroll
      for (int m = 0; m < M; ++m) part[r][m] = 0.f;
    }
    issue(i + 32);
#pragma unroll
    for (int j = 0; j < 8; ++j) {  // two bytes = four weights of every row
      float4 xv[M];
#pragma unroll
      for (int m = 0; m < M; ++m) xv[m] = xs[(m * 8 + j) * groups + i];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const uint32_t word = j < 2 ? cw[r].x : j < 4 ? cw[r].y : j < 6 ? cw[r].z : cw[r].w;
        const uint32_t h = word >> (16 * (j & 1));
        const float c0 = s_code[(h >> 4) & 15u], c1 = s_code[h & 15u];
        const float c2 = s_code[(h >> 12) & 15u], c3 = s_code[(h >> 8) & 15u];
#pragma unroll
        for (int m = 0; m < M; ++m)
          part[r][m] = fmaf(c3, xv[m].w, fmaf(c2, xv[m].z, fmaf(c1, xv[m].y, fmaf(c0, xv[m].x, part[r][m]))));
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[r][m] = fmaf(part[r][m], scale[r], acc[r][m]);
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const float v = warp_sum(acc[r][m]) * p.alpha;
      if (lane == 0 && n0 + r < p.N) {
        uint16_t* d = reinterpret_cast<uint16_t*>(p.D) + m * p.ldd + n0 + r;
        *d = static_cast<uint16_t>(q4_pack2(v, 0.f, FMT) & 0xffffu);
      }
    }
}

}  // namespace fmsb

using namespace fmsb;

constexpr int Q4V_MAX_ROWS = 4;
constexpr int Q4V_MAX_X_BYTES = 200 * 1024;  // x as fp32 in shared memory

template <int M, int FMT>
static int q4_rows_launch(const void* x, long long ldx, const Q4Params& p, cudaStream_t stream) {
  const int smem = M * p.K * 4;
  // two rows of W per warp share the reads of x; with fewer than 4096 rows that would leave SMs without a block
  const int rows = p.N >= 4096 ? 2 : 1;
  const int per_block = Q4V_WARPS * rows;
  const int grid = (p.N + per_block - 1) / per_block;
  const void* kern = rows == 2 ? (const void*)q4_rows_kernel<M, 2, FMT> : (const void*)q4_rows_kernel<M, 1, FMT>;
  if (smem > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Q4V_MAX_X_BYTES);
    if (e != cudaSuccess) return (int)e;
  }
  if (rows == 2)
    q4_rows_kernel<M, 2, FMT><<<grid, Q4V_WARPS * 32, smem, stream>>>((const uint16_t*)x, ldx, p);
  else
    q4_rows_kernel<M, 1, FMT><<<grid, Q4V_WARPS * 32, smem, stream>>>((const uint16_t*)x, ldx, p);
  return (int)cudaGetLastError();
}

template <int BN, int GPTQ>
static int q4_launch(const CUtensorMap& tx, const CUtensorMap& txa, const CUtensorMap& tbl, const Q4Params& p,
                     cudaStream_t stream) {
  static bool cfg = false;
  if (!cfg) {
    cudaError_t e = cudaFuncSetAttribute(gemm_q4_fused_kernel<BN, GPTQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Q4Cfg<BN>::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    cfg = true;
  }
  dim3 grid((p.N + BN - 1) / BN, (p.M + Q4_BM - 1) / Q4_BM);
  gemm_q4_fused_kernel<BN, GPTQ><<<grid, 64 + Q4_DQ_THREADS, Q4Cfg<BN>::kSmemBytes, stream>>>(tx, txa, tbl, p);
  return (int)cudaGetLastError();
}

static int q4_maps(CUtensorMap* tx, CUtensorMap* txa, CUtensorMap* tbl, const void* x, long long ldx, const void* xa,
                   long long ldxa, const void* bl, long long ldbl, int r2, int M, int N, int K, int bn) {
  using namespace fmsb_host;
  int rc;
  if ((rc = make_tmap_2d_16b(tx, x, M, K, ldx, 128, 64))) return rc;
  if (xa != nullptr) {
    if ((rc = make_tmap_2d_16b(txa, xa, M, r2, ldxa, 128, 64))) return rc;
    if ((rc = make_tmap_2d_16b(tbl, bl, N, r2, ldbl, bn, 64))) return rc;
  } else {
    *txa = *tx;
    *tbl = *tx;
  }
  return 0;
}

// bytes of the codes and second-level scales of a tile in shared memory
static int q4t_scale_bytes(int bn, int K) { return bn * (K / 64) + 16 + (bn * (K / 64) / 256 + 2) * 4; }

template <int BN, int FMT>
static int q4t_launch(const CUtensorMap& tx, const CUtensorMap& tw, const Q4Params& p, cudaStream_t stream) {
  const int smem = Q4tCfg<BN>::kFixed + q4t_scale_bytes(BN, p.K);
  static bool cfg = false;
  if (!cfg) {
    cudaError_t e = cudaFuncSetAttribute(gemm_q4_tma_kernel<BN, FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Q4tCfg<BN>::kFixed + Q4tCfg<BN>::kScaleBytes);
    if (e != cudaSuccess) return (int)e;
    cfg = true;
  }
  dim3 grid((p.N + BN - 1) / BN, (p.M + Q4_BM - 1) / Q4_BM);
  gemm_q4_tma_kernel<BN, FMT><<<grid, 96 + Q4T_DQ_THREADS, smem, stream>>>(tx, tw, p);
  return (int)cudaGetLastError();
}

// x [M, K] (ldx), packed shards (world pointers, shard_bytes each; world = 1: one local pointer), scales either
// `absmax` (fp32 per 64-block) or the double-quantised triple (absmax_q, code256, absmax2, offset); code16 = the
// 16-entry NF4 / FP4 table (host pointer); optional LoRA pair xa [M, R] (ldxa), bl [N, R] (ldbl), R = r2;
// y [M, N] (ldy).  K % 64 == 0, N % 8 == 0, leading dimensions % 8 == 0, bn in {32, 64, 128}
// or 0: the library chooses, the kernel for a few rows included.
extern "C" int fmsb_gemm_q4_fused(const void* x, long long ldx, void* const* packed_shards, long long shard_bytes,
                                  int world, const float* absmax, const void* absmax_q, const float* code256,
                                  const float* absmax2, float offset, const float* code16_host, const void* xa,
                                  long long ldxa, const void* bl, long long ldbl, int r2, void* y, long long ldy,
                                  float alpha, int M, int N, int K, int fmt, int bn, int* status,
                                  cudaStream_t stream) {
  using namespace fmsb_host;
  if (M <= 0 || N <= 0) return 0;
  if (K % 64 != 0 || N % 8 != 0 || (ldx % 8) || (ldy % 8) || world < 1 || world > Q4_MAX_RANKS) return -2;
  if (shard_bytes % 32 != 0 || shard_bytes * world < (long long)N * K / 2) return -2;
  if ((absmax == nullptr) == (absmax_q == nullptr)) return -2;
  if (xa != nullptr && ((ldxa % 8) || (ldbl % 8) || r2 <= 0 || bl == nullptr)) return -2;
  Q4Params p{};
  p.M = M; p.N = N; p.K = K;
  p.kblocks1 = K / 64;
  p.kblocks2 = xa != nullptr ? (r2 + 63) / 64 : 0;
  for (int i = 0; i < world; ++i) p.shard[i] = (const uint8_t*)packed_shards[i];
  p.shard_bytes = shard_bytes; p.world = world;
  p.absmax = absmax; p.absmax_q = (const uint8_t*)absmax_q; p.code256 = code256; p.absmax2 = absmax2; p.offset = offset;
  for (int i = 0; i < 16; ++i) p.code16[i] = code16_host[i];
  p.D = y; p.ldd = ldy; p.alpha = alpha; p.fmt = fmt; p.status = status;
  // Up to four rows of one local weight without a LoRA pair run on the CUDA cores (needs 16-byte aligned x and W).
  if (M <= Q4V_MAX_ROWS && bn == 0 && world == 1 && xa == nullptr && (long long)M * K * 4 <= Q4V_MAX_X_BYTES &&
      (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.shard[0]) & 15u) == 0) {
#define FMSB_Q4V(MM) \
  case MM: return fmt == 1 ? q4_rows_launch<MM, 1>(x, ldx, p, stream) : q4_rows_launch<MM, 0>(x, ldx, p, stream)
    switch (M) { FMSB_Q4V(1); FMSB_Q4V(2); FMSB_Q4V(3); FMSB_Q4V(4); }
#undef FMSB_Q4V
  }
  if (bn == 0) {
    // The tile width that keeps the busiest SM shortest: one CTA per SM, so a grid of t tiles takes ceil(t / 148)
    // turns of a time that grows with the tile's rows of W (plus a share that does not, worth about 16 rows).
    // N = 14336: 128 wide (112 tiles, one turn) instead of 64 (224, two turns); N = 4096: 32 wide, 128 tiles.
    long long best = -1;
    for (int c = 32; c <= 128; c *= 2) {
      const long long tiles = (long long)((N + c - 1) / c) * ((M + Q4_BM - 1) / Q4_BM);
      const long long cost = (tiles + 147) / 148 * (c + 16);
      if (best < 0 || cost < best) { best = cost; bn = c; }
    }
  }
  CUtensorMap tx, txa, tbl;
  if (int rc = q4_maps(&tx, &txa, &tbl, x, ldx, xa, ldxa, bl, ldbl, r2, M, N, K, bn)) return rc;
  // One local, double-quantised weight without a LoRA pair: the packed bytes by TMA (16-byte aligned; the scale codes of a
  // tile have to fit beside the stages: K up to about 15000 at 128 wide, 25000 at 64, more at 32).
  const int room = bn == 128 ? Q4tCfg<128>::kScaleBytes : bn == 64 ? Q4tCfg<64>::kScaleBytes : Q4tCfg<32>::kScaleBytes;
  if (world == 1 && xa == nullptr && absmax_q != nullptr && (reinterpret_cast<uintptr_t>(p.shard[0]) & 15u) == 0 &&
      q4t_scale_bytes(bn, K) <= room) {
    CUtensorMap tw;  // rows of K / 2 bytes, seen as K / 4 16-bit units
    if (int rc = make_tmap_2d_16b(&tw, p.shard[0], N, K / 4, K / 4, bn, 64)) return rc;
    if (bn == 128) return fmt == 1 ? q4t_launch<128, 1>(tx, tw, p, stream) : q4t_launch<128, 0>(tx, tw, p, stream);
    if (bn == 64) return fmt == 1 ? q4t_launch<64, 1>(tx, tw, p, stream) : q4t_launch<64, 0>(tx, tw, p, stream);
    if (bn == 32) return fmt == 1 ? q4t_launch<32, 1>(tx, tw, p, stream) : q4t_launch<32, 0>(tx, tw, p, stream);
    return -2;
  }
  if (bn == 128) return q4_launch<128, 0>(tx, txa, tbl, p, stream);
  if (bn == 64) return q4_launch<64, 0>(tx, txa, tbl, p, stream);
  if (bn == 32) return q4_launch<32, 0>(tx, txa, tbl, p, stream);
  return -2;
}

// GPTQ int4 form: y [M, N] = alpha * (x [M, K] . W [K, N] + xa [M, R] . bl [N, R]^T) with W given as qweight [K/8, N]
// (int32, eight k per word), scales [K/group, N] (16-bit, the format of x), qzeros [K/group, N/8] (int32) and
// zero_offset (1 for checkpoints that store the zero point minus one).  Groups follow the input features in order
// (no activation reordering) and group % 64 == 0; K % 64 == 0, N % 8 == 0; bn in {32, 64, 128}.
extern "C" int fmsb_gemm_gptq_fused(const void* x, long long ldx, const void* qweight, const void* scales,
                                    const void* qzeros, int group, int zero_offset, const void* xa, long long ldxa,
                                    const void* bl, long long ldbl, int r2, void* y, long long ldy, float alpha, int M,
                                    int N, int K, int fmt, int bn, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 64 != 0 || N % 8 != 0 || (ldx % 8) || (ldy % 8) || group <= 0 || group % 64 != 0 || K % group != 0) return -2;
  if (qweight == nullptr || scales == nullptr || qzeros == nullptr) return -2;
  if (xa != nullptr && ((ldxa % 8) || (ldbl % 8) || r2 <= 0 || bl == nullptr)) return -2;
  Q4Params p{};
  p.M = M; p.N = N; p.K = K;
  p.kblocks1 = K / 64;
  p.kblocks2 = xa != nullptr ? (r2 + 63) / 64 : 0;
  p.world = 1;
  p.gq_weight = (const uint32_t*)qweight; p.gq_scales = (const uint16_t*)scales; p.gq_zeros = (const uint32_t*)qzeros;
  p.gq_group = group; p.gq_zero_offset = zero_offset;
  p.D = y; p.ldd = ldy; p.alpha = alpha; p.fmt = fmt; p.status = status;
  CUtensorMap tx, txa, tbl;
  if (int rc = q4_maps(&tx, &txa, &tbl, x, ldx, xa, ldxa, bl, ldbl, r2, M, N, K, bn)) return rc;
  if (bn == 128) return q4_launch<128, 1>(tx, txa, tbl, p, stream);
  if (bn == 64) return q4_launch<64, 1>(tx, txa, tbl, p, stream);
  if (bn == 32) return q4_launch<32, 1>(tx, txa, tbl, p, stream);
  return -2;
}
