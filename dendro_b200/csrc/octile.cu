// Octet tiles (OctTiles, dg_internal.h): per 32 consecutive octets the distinct
// nodes of their lattices, the places of each node in the tile's 27 x 32
// lattice sums, and each lattice point's node rank.  Built on first use by an
// operator that merges a tile's sums before they leave (matvec.cu).
#include "octet.cuh"
#include "prim.cuh"

namespace dg {
namespace {

__device__ __forceinline__ int64_t gtid() { return blockIdx.x * int64_t(blockDim.x) + threadIdx.x; }
__device__ __forceinline__ int64_t gstride() { return int64_t(gridDim.x) * blockDim.x; }

constexpr int kSortKeys = 1024;  // >= kOctTileRefs, a power of two
constexpr int kBuildThreads = 256;
static_assert(kSortKeys >= kOctTileRefs, "key buffer");

// One CTA per tile: the tile's (node id, lattice position) pairs sorted in
// shared memory; a node is a run of equal ids, the positions its references.
// Nodes are ranked by falling number of references, ids ascending among
// equals, so that the k-th references of the nodes that have one are a dense
// array (refs: first the first reference of every node, then the second of
// those that have one, ...) and a warp that sums 32 nodes at a time does not
// wait for one with more references than the others.
__global__ void __launch_bounds__(kBuildThreads) octile_build(int64_t n, const uint32_t* __restrict__ oid,
                                                              uint32_t* __restrict__ ids, uint32_t* __restrict__ cnt,
                                                              uint16_t* __restrict__ hdr, uint16_t* __restrict__ refs,
                                                              uint16_t* __restrict__ lidx,
                                                              uint32_t* __restrict__ flags) {
  __shared__ uint64_t key[kSortKeys];
  __shared__ uint16_t slot[kOctTileRefs];
  __shared__ uint32_t hist[kBuildThreads / 32][kOctTileMaxRefs + 1], least[kOctTileMaxRefs + 2];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t t = blockIdx.x, o0 = t * kOctTile;
  for (int i = tid; i < kSortKeys; i += kBuildThreads) {
    uint64_t k = kNoKey;
    if (i < kOctTileRefs && o0 + i % kOctTile < n) {
      const uint32_t id = oid[int64_t(i / kOctTile) * n + o0 + i % kOctTile];
      if (id != kNoNode) k = (uint64_t(id) << 10) | uint64_t(i);
    }
    key[i] = k;
  }
  for (int i = tid; i < kOctTileRefs; i += kBuildThreads) slot[i] = 0xffffu;
  for (int i = tid; i < (kBuildThreads / 32) * (kOctTileMaxRefs + 1); i += kBuildThreads) (&hist[0][0])[i] = 0;
  __syncthreads();
  for (int k = 2; k <= kSortKeys; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int p = tid; p < kSortKeys / 2; p += kBuildThreads) {
        const int i = 2 * p - (p & (j - 1)), l = i + j;
        const uint64_t a = key[i], b = key[l];
        if ((a > b) == ((i & k) == 0)) {
          key[i] = b;
          key[l] = a;
        }
      }
      __syncthreads();
    }
  // run lengths at the runs' first entries; warp w holds entries [128 w, 128 w + 128)
  constexpr int kPer = kSortKeys / kBuildThreads;
  uint32_t len[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = w * (32 * kPer) + q * 32 + lane;
    const uint64_t id = key[i] >> 10;
    len[q] = 0;
    if (key[i] != kNoKey && (i == 0 || (key[i - 1] >> 10) != id)) {
      uint32_t c = 1;
      while (i + c < kSortKeys && (key[i + c] >> 10) == id) ++c;
      if (c > kOctTileMaxRefs) {
        atomicOr(flags, 1u);
        c = kOctTileMaxRefs;
      }
      len[q] = c;
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, len[q]);
    if (lane == __ffs(peers) - 1) hist[w][len[q]] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // first rank of each (length, warp): longer runs first
  if (tid == 0) {
    uint32_t run = 0;
    least[kOctTileMaxRefs + 1] = 0;
    for (int c = kOctTileMaxRefs; c >= 1; --c) {
      for (int v = 0; v < kBuildThreads / 32; ++v) {
        const uint32_t x = hist[v][c];
        hist[v][c] = run;
        run += x;
      }
      least[c] = run;  // nodes with at least c references
    }
    cnt[t] = run;
    atomicMax(flags + 1, run);
  }
  __syncthreads();
  if (tid < kOctTileMaxRefs) hdr[t * kOctTileMaxRefs + tid] = uint16_t(least[tid + 1]);
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = w * (32 * kPer) + q * 32 + lane;
    const uint32_t peers = __match_any_sync(0xffffffffu, len[q]);
    const uint32_t first = hist[w][len[q]];
    __syncwarp();
    if (lane == __ffs(peers) - 1) hist[w][len[q]] = first + __popc(peers);
    __syncwarp();
    if (!len[q]) continue;
    const uint32_t r = first + __popc(peers & ((1u << lane) - 1u));
    ids[t * kOctTileRefs + r] = uint32_t(key[i] >> 10);
    uint32_t off = 0;
    for (uint32_t c = 0; c < len[q]; ++c) {
      const uint32_t pos = uint32_t(key[i + c] & 1023u);
      refs[t * kOctTileRefs + off + r] = uint16_t(pos);
      slot[pos] = uint16_t(r);
      off += least[c + 1];
    }
  }
  __syncthreads();
  for (int i = tid; i < kOctTileRefs; i += kBuildThreads)
    if (o0 + i % kOctTile < n) lidx[int64_t(i / kOctTile) * n + o0 + i % kOctTile] = slot[i];
}

// Node lists of padded length (whole 16 bytes) at their places, and per node
// the number of tiles that have it.
__global__ void octile_pad(uint32_t* __restrict__ cnt, int64_t nt) {
  for (int64_t i = gtid(); i < nt; i += gstride()) cnt[i] = (cnt[i] + 3u) & ~3u;
}
__global__ void octile_lists(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ ptr,
                             const uint16_t* __restrict__ hdr, int64_t nt, uint32_t* __restrict__ nodes,
                             uint32_t* __restrict__ touch) {
  const int lane = threadIdx.x & 31;
  for (int64_t t = gtid() >> 5; t < nt; t += gstride() >> 5) {
    const uint32_t c = hdr[t * kOctTileMaxRefs];
    for (uint32_t i = lane; i < c; i += 32) {
      const uint32_t id = ids[t * kOctTileRefs + i];
      nodes[ptr[t] + i] = id;
      atomicAdd(touch + id, 1u);
    }
  }
}
__global__ void octile_mark(const uint32_t* __restrict__ ptr, const uint16_t* __restrict__ hdr, int64_t nt,
                            uint32_t* __restrict__ nodes, const uint32_t* __restrict__ touch) {
  const int lane = threadIdx.x & 31;
  for (int64_t t = gtid() >> 5; t < nt; t += gstride() >> 5) {
    const uint32_t c = hdr[t * kOctTileMaxRefs];
    for (uint32_t i = lane; i < c; i += 32) {
      const uint32_t id = nodes[ptr[t] + i];
      if (touch[id] > 1u) nodes[ptr[t] + i] = id | 0x80000000u;
    }
  }
}

// The nodes that are not in exactly one tile.
struct SharedNodes {
  const uint32_t* __restrict__ touch;
  uint32_t* __restrict__ out;
  __device__ uint32_t count(int64_t i) const { return touch[i] != 1u ? 1u : 0u; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    if (c) out[off] = uint32_t(i);
  }
};

dg_status build(dg_da* da, cudaStream_t s) {
  const OctetSet& O = da->octs;
  OctTiles& T = da->otiles;
  const int64_t n = O.n, nt = (n + kOctTile - 1) / kOctTile;
  if (da->N >= (int64_t(1) << 31)) return DG_OK;  // bit 31 of a list entry is a flag
  DBuf<uint32_t> ids, cnt, touch;
  DG_TRY(ids.alloc(nt * kOctTileRefs));
  DG_TRY(cnt.alloc(nt + 3));  // and the total, [0] flag: too many references, [1] longest list
  DG_TRY(T.hdr.alloc(nt * kOctTileMaxRefs));
  DG_TRY(T.refs.alloc(nt * kOctTileRefs));
  DG_TRY(T.lidx.alloc(27 * n));
  DG_TRY(touch.alloc(da->N));
  DG_CUDA(cudaMemsetAsync(cnt.p + nt, 0, 12, s));
  DG_CUDA(cudaMemsetAsync(touch.p, 0, 4 * da->N, s));
  octile_build<<<unsigned(nt), kBuildThreads, 0, s>>>(n, O.id.p, ids.p, cnt.p, T.hdr.p, T.refs.p, T.lidx.p,
                                                      cnt.p + nt + 1);
  octile_pad<<<grid_for(nt, 256), 256, 0, s>>>(cnt.p, nt);
  DG_CUDA(cudaGetLastError());
  DG_TRY(scan_u32(cnt.p, cnt.p, nt + 1, nullptr, s));
  uint32_t h[3];
  DG_TRY(read_words(cnt.p + nt, h, 3, s));
  if (h[1]) {  // a node that more than 16 octets of a tile list: no such mesh is known
    T.hdr.reset();
    T.refs.reset();
    T.lidx.reset();
    return DG_OK;
  }
  DG_TRY(T.nodes.alloc(h[0]));
  DG_TRY(T.ptr.alloc(nt));
  DG_CUDA(cudaMemcpyAsync(T.ptr.p, cnt.p, 4 * nt, cudaMemcpyDeviceToDevice, s));
  DG_CUDA(cudaMemsetAsync(T.nodes.p, 0, 4 * int64_t(h[0]), s));
  octile_lists<<<grid_for(nt * 32, 256), 256, 0, s>>>(ids.p, T.ptr.p, T.hdr.p, nt, T.nodes.p, touch.p);
  octile_mark<<<grid_for(nt * 32, 256), 256, 0, s>>>(T.ptr.p, T.hdr.p, nt, T.nodes.p, touch.p);
  DG_CUDA(cudaGetLastError());
  SharedNodes sf{touch.p, nullptr};
  const int64_t nb = tile_blocks(da->N);
  DBuf<uint32_t> sums;
  DG_TRY(sums.alloc(nb + 1));
  DG_TRY(tile_scan(sf, ItemCount{da->N}, sums.p, sums.p + nb, s));
  uint32_t ns = 0;
  DG_TRY(read_words(sums.p + nb, &ns, 1, s));
  DG_TRY(T.shared.alloc(ns));
  sf.out = T.shared.p;
  DG_TRY(tile_emit(sf, ItemCount{da->N}, sums.p, s));
  T.max_nodes = h[2];
  T.ntiles = nt;
  return DG_OK;
}

}  // namespace

dg_status ensure_octet_tiles(dg_da* da, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(da->tables);
  if (da->otiles.tried || !da->octs.n) return DG_OK;
  DG_TRY(build_table(s, [&](cudaStream_t t) { return build(da, t); }, [&] { da->otiles = OctTiles(); }));
  da->otiles.tried = true;
  return DG_OK;
}

}  // namespace dg
