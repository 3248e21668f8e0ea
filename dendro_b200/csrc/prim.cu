// Device-wide primitives: exclusive scan, LSD radix sort of 64-bit keys,
// adjacent-duplicate removal.  Hand-written; no CUB/Thrust on the path.
#include <cstring>
#include <utility>

#include "prim.cuh"

namespace dg {

namespace {

// Exclusive scan of nt values in place by one CTA of 1024 threads, 4
// consecutive values per thread and step; the total to *total.
__global__ void __launch_bounds__(1024) scan_small_kernel(uint32_t* __restrict__ v, int64_t nt,
                                                          uint32_t* __restrict__ total) {
  __shared__ uint32_t ws[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int64_t base = 0; base < nt; base += 4096) {
    const int64_t i0 = base + int64_t(threadIdx.x) * 4;
    uint32_t x[4], t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = i0 + k < nt ? v[i0 + k] : 0u;
      t += x[k];
    }
    const uint32_t incl = warp_incl_scan(t);
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    const uint32_t wi = warp_incl_scan(ws[lane]);  // every warp scans the 32 warp sums
    const uint32_t before = __shfl_sync(0xffffffffu, wi, w) - ws[w];
    const uint32_t sum = __shfl_sync(0xffffffffu, wi, 31);
    uint32_t run = carry + before + incl - t;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k < nt) v[i0 + k] = run;
      run += x[k];
    }
    carry += sum;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

// scan_u32 as a tile emission: every item's output is its own offset.
struct ScanItems {
  const uint32_t* in;
  uint32_t* out;
  __device__ uint32_t count(int64_t i) const { return in[i]; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t) const { out[i] = off; }
};

// ------------------------------------------------------------ radix sort --
constexpr int kRadixBits = 8;
constexpr int kBins = 1 << kRadixBits;
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;  // keys per thread (16: a third slower at 1M keys, too few CTAs)
constexpr int kSortTile = kSortThreads * kSortItems;

// A pass of the sort is three launches whatever n is: a histogram per block
// of kSortTile keys, the scan of each digit's row of block counts (a CTA per
// digit, the row total to rowtot), and the scatter, which scans the 256 row
// totals itself.  Nothing is allocated or waited for between passes; a
// device-wide scan of the whole histogram took three more launches, an
// allocation and a host wait per pass (92 passes of a mesh set-up from
// 131,072 points: 2.9 ms of kernels and most of its 46 ms of wall time).
__global__ void __launch_bounds__(kSortThreads)
radix_hist(const uint64_t* __restrict__ keys, int64_t n, int shift, uint32_t* __restrict__ hist, int nblocks) {
  __shared__ uint32_t h[kBins];
  for (int i = threadIdx.x; i < kBins; i += blockDim.x) h[i] = 0;
  __syncthreads();
  int64_t base = int64_t(blockIdx.x) * kSortTile;
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x) {
    int64_t k = base + i;
    // keys near one another often share a digit: one atomic per digit and warp
    const uint32_t d = k < n ? uint32_t((keys[k] >> shift) & (kBins - 1)) : uint32_t(kBins);
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    if (d < kBins && int(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[d], uint32_t(__popc(peers)));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kBins; i += blockDim.x) hist[int64_t(i) * nblocks + blockIdx.x] = h[i];
}

__global__ void __launch_bounds__(256) radix_rowscan(uint32_t* __restrict__ hist, int nblocks,
                                                     uint32_t* __restrict__ rowtot) {
  __shared__ uint32_t ws[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* row = hist + int64_t(blockIdx.x) * nblocks;
  uint32_t carry = 0;
  for (int base = 0; base < nblocks; base += 256) {
    const int i = base + int(threadIdx.x);
    const uint32_t x = i < nblocks ? row[i] : 0u;
    const uint32_t incl = warp_incl_scan(x);
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    uint32_t before = 0, sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      before += k < w ? ws[k] : 0u;
      sum += ws[k];
    }
    if (i < nblocks) row[i] = carry + before + incl - x;
    carry += sum;
    __syncthreads();
  }
  if (threadIdx.x == 0) rowtot[blockIdx.x] = carry;
}

// Stable scatter.  Warp w owns 32 kSortItems consecutive keys in
// slot-major, lane-minor order; ranks within the warp come from
// __match_any_sync, and per-(warp, digit) counters give the warp offsets.
__global__ void __launch_bounds__(kSortThreads)
radix_scatter(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, int64_t n, int shift,
              const uint32_t* __restrict__ offs, int nblocks, const uint32_t* __restrict__ rowtot) {
  static_assert(kBins == kSortThreads, "one thread per digit");
  __shared__ uint32_t cnt[kSortThreads / 32][kBins];
  __shared__ uint32_t wtot[kSortThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < (kSortThreads / 32) * kBins; i += blockDim.x) (&cnt[0][0])[i] = 0;
  __syncthreads();
  int64_t base = int64_t(blockIdx.x) * kSortTile + int64_t(wid) * (kSortItems * 32);
  uint64_t key[kSortItems];
  uint32_t rank[kSortItems];
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int s = 0; s < kSortItems; ++s) {
    int64_t k = base + s * 32 + lane;
    bool valid = k < n;
    key[s] = valid ? in[k] : ~0ull;
    uint32_t d = valid ? uint32_t((key[s] >> shift) & (kBins - 1)) : uint32_t(kBins);  // kBins = invalid
    uint32_t peers = __match_any_sync(0xffffffffu, d);
    uint32_t pre = (d < kBins) ? cnt[wid][d] : 0u;
    __syncwarp();
    int leader = __ffs(peers) - 1;
    if (lane == leader && d < kBins) cnt[wid][d] = pre + __popc(peers);
    __syncwarp();
    rank[s] = pre + __popc(peers & lt);
  }
  __syncthreads();
  // exclusive prefix over warps for each digit, plus the digit's first place
  // (the row totals before it) and the block's place in the digit's row
  const uint32_t rt = rowtot[threadIdx.x];
  const uint32_t rincl = warp_incl_scan(rt);
  if (lane == 31) wtot[wid] = rincl;
  __syncthreads();
  {
    const int d = threadIdx.x;
    uint32_t run = offs[int64_t(d) * nblocks + blockIdx.x] + rincl - rt;
#pragma unroll
    for (int k = 0; k < kSortThreads / 32; ++k) run += k < wid ? wtot[k] : 0u;
    for (int w = 0; w < kSortThreads / 32; ++w) {
      uint32_t c = cnt[w][d];
      cnt[w][d] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kSortItems; ++s) {
    int64_t k = base + s * 32 + lane;
    if (k < n) {
      uint32_t d = uint32_t((key[s] >> shift) & (kBins - 1));
      out[cnt[wid][d] + rank[s]] = key[s];
    }
  }
}

}  // namespace

dg_status scan_small(uint32_t* v, int64_t nt, uint32_t* total, cudaStream_t s) {
  scan_small_kernel<<<1, 1024, 0, s>>>(v, nt, total);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}

namespace {
struct HostWords {
  uint32_t* p = nullptr;
  uint32_t plain[64];
  HostWords() {
    if (cudaHostAlloc(&p, sizeof plain, cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
  }
  ~HostWords() {
    if (p) cudaFreeHost(p);
  }
};
}  // namespace

dg_status read_words(const uint32_t* dev, uint32_t* host, int nw, cudaStream_t s) {
  static thread_local HostWords w;
  DG_CHECK(nw > 0 && nw <= 64, DG_EINVAL, "read_words: at most 64 words");
  uint32_t* at = w.p ? w.p : w.plain;
  DG_CUDA(cudaMemcpyAsync(at, dev, sizeof(uint32_t) * size_t(nw), cudaMemcpyDeviceToHost, s));
  DG_CUDA(cudaStreamSynchronize(s));
  memcpy(host, at, sizeof(uint32_t) * size_t(nw));
  return DG_OK;
}

dg_status scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* total, cudaStream_t s) {
  if (n <= 0) {
    if (total) *total = 0;
    return DG_OK;
  }
  DG_CHECK(n < (int64_t(1) << 31), DG_EINVAL, "scan: too many elements");
  const int64_t nb = tile_blocks(n);
  DBuf<uint32_t> sums;
  DG_TRY(sums.alloc(nb + 1));
  const ScanItems f{in, out};
  const ItemCount nc{n};
  DG_TRY(tile_scan(f, nc, sums.p, sums.p + nb, s));
  DG_TRY(tile_emit(f, nc, sums.p, s));
  if (total) DG_TRY(read_words(sums.p + nb, total, 1, s));
  return DG_OK;
}

dg_status radix_sort_u64(DBuf<uint64_t>& keys, DBuf<uint64_t>& tmp, int64_t n, int bits, cudaStream_t s,
                         int start_bit) {
  if (n <= 1) return DG_OK;
  DG_CHECK(n < (int64_t(1) << 31), DG_EINVAL, "radix sort: too many keys");
  const int nblocks = int((n + kSortTile - 1) / kSortTile);
  DBuf<uint32_t> hist;
  DG_TRY(hist.alloc(int64_t(kBins) * nblocks + kBins));
  uint32_t* rowtot = hist.p + int64_t(kBins) * nblocks;
  const int passes = (bits + kRadixBits - 1) / kRadixBits;
  for (int p = 0; p < passes; ++p) {
    const int shift = start_bit + p * kRadixBits;
    radix_hist<<<nblocks, kSortThreads, 0, s>>>(keys.p, n, shift, hist.p, nblocks);
    radix_rowscan<<<kBins, 256, 0, s>>>(hist.p, nblocks, rowtot);
    radix_scatter<<<nblocks, kSortThreads, 0, s>>>(keys.p, tmp.p, n, shift, hist.p, nblocks, rowtot);
    std::swap(keys, tmp);
  }
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}

dg_status unique_u64(DBuf<uint64_t>& keys, DBuf<uint64_t>& tmp, int64_t n, int64_t* n_out, cudaStream_t s) {
  *n_out = n;
  if (n <= 1) return DG_OK;
  const int64_t nb = tile_blocks(n);
  DBuf<uint32_t> sums;
  DG_TRY(sums.alloc(nb + 1));
  const UniqueKeys f{keys.p, tmp.p};
  const ItemCount nc{n};
  DG_TRY(tile_scan(f, nc, sums.p, sums.p + nb, s));
  DG_TRY(tile_emit(f, nc, sums.p, s));
  uint32_t total = 0;
  DG_TRY(read_words(sums.p + nb, &total, 1, s));
  std::swap(keys, tmp);
  *n_out = total;
  return DG_OK;
}

}  // namespace dg
