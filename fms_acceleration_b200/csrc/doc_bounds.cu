// Document bounds of a packed batch from its position ids, on the device.
//
// A new document starts wherever the position is 0: start[t] = the last such index up to t, end[t] = the next one after t
// (or T).  Tokens before the first 0 belong to the first document, as in the searchsorted form of this rule: their
// start is the first 0 (T when there is none) and their end the 0 after it.  Finding the starts with torch.nonzero copied
// their number to the host, so every forward waited for the device to run dry and the whole step was enqueued behind an
// idle GPU (1 ms of a 6 ms two-layer step); this is one launch that also narrows the positions to 32 bits.
//
// One CTA per 1024 tokens.  The first launch notes the first and the last start of every tile; the second finds the start that
// reaches into a tile and the one that ends it from those notes, 1024 tiles a step, and the rest within the tile.  Tokens
// before the first 0 also need the start after it: the CTA looks for that one too, once.  Searching the positions
// themselves, tile by tile, and letting every token before the first 0 walk through the next document by itself took
// 5629 us for 1000 such tokens before a document of 64536 and 2458 us for one document of 2^20 tokens; this form 38 and
// 117 us (a call, host included).
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

// tiles[i] = (first start in tile i or T, last one or -1)
template <typename I>
__global__ void __launch_bounds__(DB_T) doc_tiles_kernel(const I* __restrict__ pos, int2* __restrict__ tiles, int T) {
  __shared__ int red[32];
  const int t = blockIdx.x * DB_T + threadIdx.x;
  const bool zero = t < T && pos[t] == 0;
  const int first = T - db_block_max(zero ? T - t : 0, red), last = db_block_max(zero ? t : -1, red);
  if (threadIdx.x == 0) tiles[blockIdx.x] = make_int2(first, last);
}

// first start in the tiles from `lo` on, T if there is none; the whole CTA calls it with the same arguments
__device__ __forceinline__ int db_first_from(const int2* __restrict__ tiles, int lo, int n, int T, int* red) {
  for (; lo < n; lo += DB_T) {
    const int i = lo + threadIdx.x;
    const int r = db_block_max(i < n ? T - tiles[i].x : 0, red);
    if (r > 0) return T - r;
  }
  return T;
}

template <typename I>
__global__ void __launch_bounds__(DB_T) doc_bounds_kernel(const I* __restrict__ pos, const int2* __restrict__ tiles,
                                                          int* __restrict__ pos32, int* __restrict__ start,
                                                          int* __restrict__ end, int T) {
  __shared__ int red[32], wmax[32], wmin[32], lead;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = gridDim.x;
  const int t = blockIdx.x * DB_T + threadIdx.x;
  const I v = t < T ? pos[t] : (I)1;
  if (t < T) pos32[t] = (int)v;
  const bool zero = t < T && v == 0;
  // the last start before this tile, and the first one after it
  int before = -1;
  for (int hi = blockIdx.x; hi > 0 && before < 0; hi -= DB_T) {
    const int i = hi - 1 - (int)threadIdx.x;
    before = db_block_max(i >= 0 ? tiles[i].y : -1, red);
  }
  const int after = db_first_from(tiles, blockIdx.x + 1, n, T, red);
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
  // tokens before the first start are the first ones of their tile and share both bounds: that start and the next one
  if (threadIdx.x == 0) lead = s < 0 ? nxt : -1;
  __syncthreads();
  if (lead >= 0) {
    int second = T;
    if (lead < T) {
      const int tile = lead / DB_T, u = tile * DB_T + threadIdx.x;
      const int r = db_block_max(u > lead && u < T && pos[u] == 0 ? T - u : 0, red);
      second = r > 0 ? T - r : db_first_from(tiles, tile + 1, n, T, red);
    }
    if (s < 0) {
      s = lead;
      nxt = second;
    }
  }
  if (t >= T) return;
  start[t] = s;
  end[t] = nxt;
}

template <typename I>
static void doc_bounds(const I* pos, int* pos32, int* start, int* end, int* tiles, int T, cudaStream_t stream) {
  const int blocks = (T + DB_T - 1) / DB_T;
  // a single tile has no neighbours to look at
  if (blocks > 1) doc_tiles_kernel<I><<<blocks, DB_T, 0, stream>>>(pos, (int2*)tiles, T);
  doc_bounds_kernel<I><<<blocks, DB_T, 0, stream>>>(pos, (const int2*)tiles, pos32, start, end, T);
}

}  // namespace fmsb

// pos [T] int64 (wide = 1) or int32; pos32, start, end [T] int32; tiles: scratch of 2 ceil(T / 1024) ints, 8-byte aligned.
extern "C" int fmsb_doc_bounds(const void* pos, int wide, int* pos32, int* start, int* end, int* tiles, int T,
                               cudaStream_t stream) {
  using namespace fmsb;
  if (T <= 0) return 0;
  if (T > 0x7fffffff - DB_T || (reinterpret_cast<uintptr_t>(tiles) & 7u) != 0) return -2;  // indexes run past T by up to a tile
  if (wide) doc_bounds((const long long*)pos, pos32, start, end, tiles, T, stream);
  else doc_bounds((const int*)pos, pos32, start, end, tiles, T, stream);
  return (int)cudaGetLastError();
}
