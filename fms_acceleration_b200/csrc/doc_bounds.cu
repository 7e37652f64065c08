// Document bounds of a packed batch from its position ids, on the device.
//
// A new document starts wherever the position is 0: start[t] = the last such index up to t, end[t] = the next one after t
// (or T).  Tokens before the first 0 belong to the first document, as in the searchsorted form of this rule: their
// start is the first 0 (T when there is none) and their end the 0 after it.  Finding the starts with torch.nonzero copied
// their number to the host, so every forward waited for the device to run dry and the whole step was enqueued behind an
// idle GPU (1 ms of a 6 ms two-layer step); this is one launch that also narrows the positions to 32 bits.
//
// One CTA per 1024 tokens; it finds the start that reaches into it and the one that ends it by searching outwards, tile by
// tile, so no CTA waits for another.  The search is as long as the documents are.
#include "common.cuh"

namespace fmsb {

constexpr int DB_T = 1024;

__device__ __forceinline__ int db_block_max(int v, int* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  v = red[lane];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <typename I>
__global__ void __launch_bounds__(DB_T) doc_bounds_kernel(const I* __restrict__ pos, int* __restrict__ pos32,
                                                          int* __restrict__ start, int* __restrict__ end, int T) {
  __shared__ int red[32], wmax[32], wmin[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b0 = blockIdx.x * DB_T, t = b0 + threadIdx.x;
  const I v = t < T ? pos[t] : (I)1;
  if (t < T) pos32[t] = (int)v;
  const bool zero = t < T && v == 0;
  // the last start before this tile, and the first one after it
  int before = -1, after = T;
  for (int base = b0 - DB_T; base >= 0 && before < 0; base -= DB_T)
    before = db_block_max(pos[base + threadIdx.x] == 0 ? base + (int)threadIdx.x : -1, red);
  for (int base = b0 + DB_T; base < T && after == T; base += DB_T) {
    const int u = base + threadIdx.x;
    after = T - max(0, db_block_max(u < T && pos[u] == 0 ? T - u : 0, red));
  }
  // inclusive maximum of the starts up to t, minimum of those after t
  int s = zero ? t : -1, e = zero ? t : T;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, s, o), b = __shfl_down_sync(0xffffffffu, e, o);
    if (lane >= o) s = max(s, a);
    if (lane + o < 32) e = min(e, b);
  }
  __syncthreads();
  if (lane == 31) wmax[warp] = s;
  if (lane == 0) wmin[warp] = e;
  __syncthreads();
  int nxt = __shfl_down_sync(0xffffffffu, e, 1);  // exclusive: starts after t
  if (lane == 31) nxt = T;
  for (int w = 0; w < warp; ++w) s = max(s, wmax[w]);
  for (int w = warp + 1; w < 32; ++w) nxt = min(nxt, wmin[w]);
  s = max(s, before);
  nxt = min(nxt, after);
  if (t >= T) return;
  if (s < 0) {  // before the first start: the first document
    s = nxt;
    int u = nxt + 1;
    while (u < T && pos[u] != 0) ++u;
    nxt = min(u, T);
  }
  start[t] = s;
  end[t] = nxt;
}

}  // namespace fmsb

// pos [T] int64 (wide = 1) or int32; pos32, start, end [T] int32.
extern "C" int fmsb_doc_bounds(const void* pos, int wide, int* pos32, int* start, int* end, int T, cudaStream_t stream) {
  using namespace fmsb;
  if (T <= 0) return 0;
  const int blocks = (T + DB_T - 1) / DB_T;
  if (wide) doc_bounds_kernel<long long><<<blocks, DB_T, 0, stream>>>((const long long*)pos, pos32, start, end, T);
  else doc_bounds_kernel<int><<<blocks, DB_T, 0, stream>>>((const int*)pos, pos32, start, end, T);
  return (int)cudaGetLastError();
}
