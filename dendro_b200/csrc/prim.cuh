// Tile-wise count / scan / emit over n items, n known on the host or only on
// the device.  A tile is kTileItems consecutive items of one CTA; count()
// gives an item's number of outputs, emit(i, off, c) writes them from output
// off on.  Three launches (tile sums, one CTA that scans the sums, tiles
// again), no allocation besides the caller's sums array and no
// synchronisation: the total stays on the device until the caller asks.
#pragma once

#include "dg_internal.h"

namespace dg {

// Number of items: host, or *dev + add when dev is set (host is then a bound).
struct ItemCount {
  int64_t host = 0;
  const uint32_t* dev = nullptr;
  uint32_t add = 0;
  __device__ __forceinline__ int64_t get() const {
    if (!dev) return host;
    const int64_t n = int64_t(*dev) + add;
    return n < host ? n : host;
  }
};

constexpr int kTileThreads = 256;
constexpr int kTilePer = 8;  // items per lane: 8 consecutive groups of 32 per warp
constexpr int kTileItems = kTileThreads * kTilePer;
inline int64_t tile_blocks(int64_t n) { return n > 0 ? (n + kTileItems - 1) / kTileItems : 1; }

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

template <class F>
__global__ void __launch_bounds__(kTileThreads) tile_count_kernel(F f, ItemCount nc, uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[kTileThreads / 32];
  const int64_t n = nc.get();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t base = int64_t(blockIdx.x) * kTileItems + w * (32 * kTilePer) + lane;
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kTilePer; ++k) {
    const int64_t i = base + 32 * k;
    if (i < n) s += f.count(i);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) ws[w] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
#pragma unroll
    for (int i = 0; i < kTileThreads / 32; ++i) t += ws[i];
    sums[blockIdx.x] = t;
  }
}

template <class F>
__global__ void __launch_bounds__(kTileThreads) tile_emit_kernel(F f, ItemCount nc, const uint32_t* __restrict__ sums) {
  __shared__ uint32_t ws[kTileThreads / 32];
  const int64_t n = nc.get();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t base = int64_t(blockIdx.x) * kTileItems + w * (32 * kTilePer) + lane;
  if (int64_t(blockIdx.x) * kTileItems >= n) return;
  uint32_t c[kTilePer], off[kTilePer], run = 0;
#pragma unroll
  for (int k = 0; k < kTilePer; ++k) {
    const int64_t i = base + 32 * k;
    c[k] = i < n ? f.count(i) : 0u;
    const uint32_t incl = warp_incl_scan(c[k]);
    off[k] = run + incl - c[k];
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) ws[w] = run;
  __syncthreads();
  uint32_t start = sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kTileThreads / 32; ++i) start += i < w ? ws[i] : 0u;
#pragma unroll
  for (int k = 0; k < kTilePer; ++k) {
    const int64_t i = base + 32 * k;
    if (i < n) f.emit(i, start + off[k], c[k]);
  }
}

// Exclusive scan of nt values in place by one CTA; the total to *total (device).
dg_status scan_small(uint32_t* v, int64_t nt, uint32_t* total, cudaStream_t s);

// The sums of f's tiles, scanned: sums holds tile_blocks(n.host) values, the
// total goes to *total on the device.
template <class F>
dg_status tile_scan(const F& f, const ItemCount& n, uint32_t* sums, uint32_t* total, cudaStream_t s) {
  const int64_t nb = tile_blocks(n.host);
  tile_count_kernel<F><<<unsigned(nb), kTileThreads, 0, s>>>(f, n, sums);
  DG_CUDA(cudaGetLastError());
  return scan_small(sums, nb, total, s);
}
// The outputs of f after tile_scan.
template <class F>
dg_status tile_emit(const F& f, const ItemCount& n, const uint32_t* sums, cudaStream_t s) {
  tile_emit_kernel<F><<<unsigned(tile_blocks(n.host)), kTileThreads, 0, s>>>(f, n, sums);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}

// Adjacent duplicates of a sorted key array dropped.
struct UniqueKeys {
  const uint64_t* __restrict__ in;
  uint64_t* __restrict__ out;
  __device__ uint32_t count(int64_t i) const { return i == 0 || in[i] != in[i - 1] ? 1u : 0u; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    if (c) out[off] = in[i];
  }
};

// First i in [lo, n) with a[i] >= key, searched outwards from lo (the answer
// is expected near lo): doubling steps, then bisection of the last step.
__device__ __forceinline__ int64_t gallop(const uint64_t* __restrict__ a, int64_t lo, int64_t n, uint64_t key) {
  int64_t hi = lo, step = 1;
  while (hi < n && a[hi] < key) {
    lo = hi + 1;
    hi += step;
    step <<= 1;
  }
  if (hi > n) hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Open-addressing hash of 64-bit keys (never all ones), linear probing, a
// power of two of slots: the slot is the top bits of the key multiplied by odd
// constants (2^64 over the golden ratio) twice, the halves folded between --
// with one multiplication the regular keys of a cloud's octants run into long
// probe sequences (building the map took twice as long), and a range reduction
// by a 128-bit product made the kernels bound by integer arithmetic.
constexpr uint64_t kNoKey = ~0ull;
constexpr int kMaxProbes = 512;  // an insertion that probes further reports a full table
struct HashShape {
  uint32_t shift;  // 64 - log2(slots)
  __host__ __device__ uint64_t slots() const { return 1ull << (64u - shift); }
};
inline HashShape hash_shape(int64_t entries) {  // at most half full
  uint32_t b = 4;
  while ((int64_t(1) << b) < 2 * entries) ++b;
  return HashShape{64u - b};
}
__device__ __forceinline__ uint64_t hash_mix(uint64_t key) {
  key *= 0x9e3779b97f4a7c15ull;
  key ^= key >> 32;
  return key * 0x9e3779b97f4a7c15ull;
}
// 31 bits of the mixed key below the slot's
__device__ __forceinline__ uint32_t hash_tag(uint64_t mix, HashShape H) {
  return uint32_t(mix >> (H.shift - 31u)) & 0x7fffffffu;
}

// Steps between cells in Morton order without taking coordinates apart: a
// coordinate's bits sit at every third place, so adding with the other places
// filled by ones carries from one of its bits to the next.  `unit` is the
// coordinate's bit of the step; leaving the domain [0, 2^D) on a positive side
// sets a bit at or above 3 D, so does leaving it on a negative one.
__device__ __forceinline__ uint64_t axis_bits(int a) { return 0x1249249249249249ull << a; }
__device__ __forceinline__ uint64_t morton_inc(uint64_t m, int a, uint64_t unit) {
  const uint64_t A = axis_bits(a);
  return (((m | ~A) + unit) & A) | (m & ~A);
}
__device__ __forceinline__ uint64_t morton_dec(uint64_t m, int a, uint64_t unit) {
  const uint64_t A = axis_bits(a);
  return (((m & A) - unit) & A) | (m & ~A);
}

// Copies nw device words to the host and waits for the stream (a page-locked
// buffer per thread; at most 64 words).
dg_status read_words(const uint32_t* dev, uint32_t* host, int nw, cudaStream_t s);

}  // namespace dg
