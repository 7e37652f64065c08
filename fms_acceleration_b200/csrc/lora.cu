// Packing and unpacking of the LoRA factors of a projection group (q|k|v, gate|up, o, down).
//
// The group's low-rank update rides in its GEMM as one operand pair, so the B factors are laid out block-diagonally with the
// scaling folded in, and the gradients of that layout are cut apart again.  With torch operators that was a zero fill and
// three launches per adapter in the forward, three more per adapter in the backward: some forty launches of a few
// microseconds in a two-layer QLoRA step, one per group and direction here.
#include "common.cuh"

namespace fmsb {

constexpr int kLoraMax = 8;

struct LoraGroup {
  const void* b[kLoraMax];  // [out, r] (pack)
  void* ga[kLoraMax];       // [r, in] (unpack; null: skip)
  void* gb[kLoraMax];       // [out, r]
  float s[kLoraMax];
  int o0[kLoraMax], o1[kLoraMax];  // rows of the group's output
  int r0[kLoraMax], r1[kLoraMax];  // columns of the packed rank
  int n, rp;
};

// blk [total_out, rp]: blk[o0 + i, r0 + j] = round(s * b[i, j]), zero elsewhere
template <typename T>
__global__ void __launch_bounds__(256) lora_pack_kernel(const __grid_constant__ LoraGroup g, T* __restrict__ blk, long long total) {
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= total) return;
  const int row = (int)(i / g.rp), col = (int)(i % g.rp);
  float v = 0.f;
#pragma unroll
  for (int a = 0; a < kLoraMax; ++a)
    if (a < g.n && row >= g.o0[a] && row < g.o1[a] && col >= g.r0[a] && col < g.r1[a])
      v = g.s[a] * (float)reinterpret_cast<const T*>(g.b[a])[(long long)(row - g.o0[a]) * (g.r1[a] - g.r0[a]) + col - g.r0[a]];
  blk[i] = (T)v;
}

// ga = round(da[r0:r1]), gb = round(s * db[o0:o1, r0:r1]); da [rp, in], db [total_out, rp] fp32.  grid.y = adapter.
template <typename T>
__global__ void __launch_bounds__(256) lora_unpack_kernel(const __grid_constant__ LoraGroup g, const float* __restrict__ da,
                                                          const float* __restrict__ db, int in) {
  const int a = blockIdx.y, r = g.r1[a] - g.r0[a], out = g.o1[a] - g.o0[a];
  const long long na = (long long)r * in, total = na + (long long)out * r;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    if (i < na) {
      reinterpret_cast<T*>(g.ga[a])[i] = (T)da[(long long)g.r0[a] * in + i];
    } else {
      const long long j = i - na;
      const int row = (int)(j / r), col = (int)(j % r);
      reinterpret_cast<T*>(g.gb[a])[j] = (T)(db[(long long)(g.o0[a] + row) * g.rp + g.r0[a] + col] * g.s[a]);
    }
  }
}

}  // namespace fmsb

using namespace fmsb;

// desc: per adapter (o0, o1, r0, r1); s: scalings; all host arrays of n.
static bool lora_group(LoraGroup& g, int n, const int* desc, const float* s, int rp) {
  if (n < 1 || n > kLoraMax || rp <= 0) return false;
  g = LoraGroup{};
  g.n = n;
  g.rp = rp;
  for (int a = 0; a < n; ++a) {
    g.o0[a] = desc[4 * a]; g.o1[a] = desc[4 * a + 1]; g.r0[a] = desc[4 * a + 2]; g.r1[a] = desc[4 * a + 3];
    g.s[a] = s[a];
    if (g.o0[a] < 0 || g.o1[a] < g.o0[a] || g.r0[a] < 0 || g.r1[a] <= g.r0[a] || g.r1[a] > rp) return false;
  }
  return true;
}

extern "C" int fmsb_lora_pack(int n, void* const* b, const int* desc, const float* s, void* blk, int total_out, int rp, int dtype,
                              cudaStream_t stream) {
  LoraGroup g;
  if (!lora_group(g, n, desc, s, rp)) return -2;
  for (int a = 0; a < n; ++a) g.b[a] = b[a];
  const long long total = (long long)total_out * rp;
  if (total <= 0) return 0;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (dtype == 1) lora_pack_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(g, (__nv_bfloat16*)blk, total);
  else if (dtype == 0) lora_pack_kernel<__half><<<blocks, 256, 0, stream>>>(g, (__half*)blk, total);
  else return -2;
  return (int)cudaGetLastError();
}

extern "C" int fmsb_lora_unpack(int n, void* const* ga, void* const* gb, const int* desc, const float* s, const float* da,
                                const float* db, int in, int rp, int dtype, cudaStream_t stream) {
  LoraGroup g;
  if (in <= 0 || !lora_group(g, n, desc, s, rp)) return -2;
  long long most = 0;
  for (int a = 0; a < n; ++a) {
    g.ga[a] = ga[a];
    g.gb[a] = gb[a];
    const long long t = (long long)(g.r1[a] - g.r0[a]) * (in + g.o1[a] - g.o0[a]);
    if (t > most) most = t;
  }
  long long blocks = (most + 255) / 256;
  if (blocks > 1184) blocks = 1184;
  const dim3 grid((unsigned)blocks, n);
  if (dtype == 1) lora_unpack_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(g, da, db, in);
  else if (dtype == 0) lora_unpack_kernel<__half><<<grid, 256, 0, stream>>>(g, da, db, in);
  else return -2;
  return (int)cudaGetLastError();
}
