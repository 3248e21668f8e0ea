// Octree construction on the GPU: points -> linear octree (points2OctreeSeq /
// p2oLocal, src/oct/Construct.C:880-1015), 2:1 balance with corners
// (balanceOctree -> comboRipple, src/oct/Balance.C:31,767,1162) and one level
// of coarsening (coarsenOctree, src/oct/Coarsen.C:53-104).
//
// All three are integer key manipulations on Morton keys: sort, adjacent
// unique, a hash set and per-key arithmetic.  Outputs are bit-exact with the
// reference's octant lists (anchors and levels, Morton order).  Counts stay on
// the device; each operation reads one of them back, to size its output.
#include <algorithm>

#include "prim.cuh"

namespace dg {

namespace {

__device__ __forceinline__ int64_t gtid() { return blockIdx.x * int64_t(blockDim.x) + threadIdx.x; }
__device__ __forceinline__ int64_t gstride() { return int64_t(gridDim.x) * blockDim.x; }

// --------------------------------------------------------------- points --
// Construct.C:897-911: px = (uint)(x * 2^D / gLen) with gLen = 1.
__global__ void quantise_points(const double* __restrict__ pts, int64_t n, uint32_t D,
                                uint64_t* __restrict__ keys, uint32_t* __restrict__ bad) {
  const double scale = double(1u << D);
  const uint32_t top = 1u << D;
  for (int64_t i = gtid(); i < n; i += gstride()) {
    double vx = pts[3 * i] * scale / 1.0, vy = pts[3 * i + 1] * scale / 1.0, vz = pts[3 * i + 2] * scale / 1.0;
    if (!(vx >= 0.0 && vy >= 0.0 && vz >= 0.0 && vx < double(top) && vy < double(top) && vz < double(top))) {
      atomicExch(bad, 1u);
      vx = vy = vz = 0.0;
    }
    keys[i] = morton(uint32_t(vx), uint32_t(vy), uint32_t(vz));
  }
}

__device__ __forceinline__ uint32_t common_level(uint64_t a, uint64_t b, uint32_t D) {
  uint64_t x = a ^ b;
  if (!x) return D;
  uint32_t lz = uint32_t(__clzll(x)) - (64u - 3u * D);
  return lz / 3u;
}

// Leaf of each sorted point: the octant at level l containing point i is
// split iff some window of m+1 consecutive points holding i lies inside it,
// i.e. iff keys j and j+m share the level-l prefix.  The leaf is one level
// below the deepest split ancestor (never deeper than D).
__global__ void point_leaves(const uint64_t* __restrict__ pk, int64_t n, uint32_t D, uint32_t m,
                             uint64_t* __restrict__ leaf) {
  for (int64_t i = gtid(); i < n; i += gstride()) {
    int64_t lo = i - int64_t(m) > 0 ? i - int64_t(m) : 0;
    int64_t hi = i < n - 1 - int64_t(m) ? i : n - 1 - int64_t(m);
    uint32_t best = 0;
    for (int64_t j = lo; j <= hi; ++j) {
      uint32_t c = common_level(pk[j], pk[j + m], D);
      c = c < D - 1 ? c : D - 1;
      best = c > best ? c : best;
    }
    uint32_t L = best + 1;
    uint64_t anchor = pk[i] & ~((1ull << (3u * (D - L))) - 1ull);
    leaf[i] = okey(anchor, L);
  }
}

// Number of maximal aligned octants covering the Morton cell range [lo, hi).
__device__ __forceinline__ uint32_t gap_blocks(uint64_t lo, uint64_t hi, uint32_t D, uint64_t* out) {
  uint32_t c = 0;
  while (lo < hi) {
    uint32_t k = lo ? (uint32_t(__ffsll(lo)) - 1u) / 3u : D;
    if (k > D) k = D;
    uint64_t span = hi - lo;
    while (k > 0 && (1ull << (3u * k)) > span) --k;
    if (out) out[c] = okey(lo, D - k);
    ++c;
    lo += 1ull << (3u * k);
  }
  return c;
}

__device__ __forceinline__ void gap_bounds(const uint64_t* __restrict__ lk, int64_t u, int64_t k, uint32_t D,
                                           uint64_t& lo, uint64_t& hi) {
  if (k == 0) {
    lo = 0;
  } else {
    uint64_t p = lk[k - 1];
    lo = okey_m(p) + (1ull << (3u * (D - okey_l(p))));
  }
  hi = (k == u) ? (1ull << (3u * D)) : okey_m(lk[k]);
}

// Item k of u + 1: the octants of the gap before leaf k, then the leaf.
struct Gaps {
  const uint64_t* __restrict__ lk;
  const uint32_t* __restrict__ nu;  // number of leaves u
  uint32_t D;
  uint64_t* __restrict__ out;
  __device__ uint32_t count(int64_t k) const {
    const int64_t u = *nu;
    uint64_t lo, hi;
    gap_bounds(lk, u, k, D, lo, hi);
    return gap_blocks(lo, hi, D, nullptr) + (k < u ? 1u : 0u);
  }
  __device__ void emit(int64_t k, uint32_t off, uint32_t) const {
    const int64_t u = *nu;
    uint64_t lo, hi;
    gap_bounds(lk, u, k, D, lo, hi);
    const uint32_t c = gap_blocks(lo, hi, D, out + off);
    if (k < u) out[off + c] = lk[k];
  }
};

// -------------------------------------------------------------- balance --
// The internal octants U of the balanced octree, as a set: the parents of the
// input's leaves, and for every internal octant u at level l the parents of
// its 26 neighbours of level l (an internal octant's neighbours must exist, so
// their parents are internal).  Along an axis those are u's parent and the
// parent's neighbour on u's side of it, so 8 cells at level l - 1 and not 27
// octants at level l, which halves and more what is looked up; the set is a
// hash table, because sorting each level's candidates (8 passes over 27 keys
// per internal octant) was two thirds of the kernel time.  Levels are worked
// from the finest up, one launch each, with all counts on the device.
struct InternalSet {
  uint64_t* table;     // okeys, kNoKey empty
  HashShape shape;
  uint64_t* list;      // [lcap] the set's members in order of insertion
  uint32_t lcap;
  uint32_t* count;     // [0] members from leaves, [1] flag: table or list full, [2 + l] members of level l added
                       // below leaves' parents
};

// Whether the key is new to the set; a full table raises the flag.  `h` is the
// key's slot and `cur` what the caller read there (reads of several keys
// overlap).
__device__ __forceinline__ uint64_t set_slot(const InternalSet& S, uint64_t key) {
  return hash_mix(key) >> S.shape.shift;
}
__device__ __forceinline__ uint64_t set_peek(const InternalSet& S, uint64_t h) {
  return *reinterpret_cast<volatile uint64_t*>(S.table + h);
}
__device__ __forceinline__ bool set_insert(const InternalSet& S, uint64_t key, uint64_t h, uint64_t cur) {
  const uint64_t wrap = S.shape.slots() - 1;
  for (int probe = 0; probe < kMaxProbes; ++probe) {
    if (cur == kNoKey) cur = atomicCAS(reinterpret_cast<unsigned long long*>(S.table + h), kNoKey, key);
    if (cur == kNoKey) return true;
    if (cur == key) return false;
    h = (h + 1) & wrap;
    cur = set_peek(S, h);
  }
  S.count[1] = 1u;
  return false;
}

// The CTA's new keys behind the first `base` members, counted in *ctr: one
// atomic per kSetItems items of every thread.  (One per warp and item, all on
// the same address, took most of the 125 us that the 3M leaves of the 1M-point
// benchmark octree did: 94K atomics.)  All threads of
// the CTA call it.
constexpr int kSetThreads = 256;
constexpr int kSetItems = 2;
__device__ __forceinline__ void set_append(const InternalSet& S, const bool (&is_new)[kSetItems],
                                           const uint64_t (&key)[kSetItems], uint32_t base, uint32_t* ctr) {
  __shared__ uint32_t ws[kSetThreads / 32], at0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t mine = 0;
#pragma unroll
  for (int k = 0; k < kSetItems; ++k) mine += is_new[k];
  const uint32_t incl = warp_incl_scan(mine);
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  uint32_t before = 0, sum = 0;
#pragma unroll
  for (int k = 0; k < kSetThreads / 32; ++k) {
    before += k < w ? ws[k] : 0u;
    sum += ws[k];
  }
  if (threadIdx.x == 0 && sum) at0 = atomicAdd(ctr, sum);
  __syncthreads();
  uint32_t at = base + at0 + before + incl - mine;
#pragma unroll
  for (int k = 0; k < kSetItems; ++k) {
    if (!is_new[k]) continue;
    if (at < S.lcap) S.list[at] = key[k];
    else S.count[1] = 1u;
    ++at;
  }
}

__device__ __forceinline__ uint64_t parent_key(uint64_t ok, uint32_t D) {
  uint32_t l = okey_l(ok);
  uint32_t pl = l ? l - 1 : 0;
  uint64_t m = okey_m(ok) & ~((1ull << (3u * (D - pl))) - 1ull);
  return okey(m, pl);
}

__global__ void __launch_bounds__(kSetThreads) balance_leaf_parents(const uint64_t* __restrict__ leaf, int64_t n,
                                                                    uint32_t D, InternalSet S) {
  constexpr int64_t kStep = kSetThreads * kSetItems;
  for (int64_t i0 = int64_t(blockIdx.x) * kStep; i0 < n; i0 += int64_t(gridDim.x) * kStep) {
    bool fresh[kSetItems];
    uint64_t pk[kSetItems];
#pragma unroll
    for (int k = 0; k < kSetItems; ++k) {
      const int64_t i = i0 + k * kSetThreads + threadIdx.x;
      fresh[k] = false;
      pk[k] = 0;
      if (i < n && okey_l(leaf[i]) > 0) {
        pk[k] = parent_key(leaf[i], D);
        // siblings are mostly adjacent: only the first of a run inserts
        if (i == 0 || okey_l(leaf[i - 1]) == 0 || parent_key(leaf[i - 1], D) != pk[k]) {
          const uint64_t h = set_slot(S, pk[k]);
          fresh[k] = set_insert(S, pk[k], h, set_peek(S, h));
        }
      }
    }
    set_append(S, fresh, pk, 0u, S.count);
  }
}

// The members of level l (those among the leaves' parents, and those that the
// level below added) add theirs at level l - 1; 8 lanes per member.
__global__ void __launch_bounds__(kSetThreads) balance_level(uint32_t l, uint32_t D, InternalSet S) {
  constexpr int64_t kStep = kSetThreads * kSetItems;
  const uint32_t n0 = min(S.count[0], S.lcap);
  uint32_t base = n0;
  for (uint32_t k = l + 1; k < D; ++k) base += S.count[2 + k];
  const uint32_t nl = S.count[2 + l];
  const uint32_t wbase = base + nl;
  const int64_t items = (int64_t(n0) + nl) * 8;
  for (int64_t t0 = int64_t(blockIdx.x) * kStep; t0 < items; t0 += int64_t(gridDim.x) * kStep) {
    bool fresh[kSetItems], mine[kSetItems];
    uint64_t key[kSetItems], h[kSetItems], cur[kSetItems];
    bool any = false;
#pragma unroll
    for (int k = 0; k < kSetItems; ++k) {
      const int64_t t = t0 + k * kSetThreads + threadIdx.x;
      fresh[k] = mine[k] = false;
      key[k] = h[k] = cur[k] = 0;
      if (t >= items) continue;
      const uint32_t j = uint32_t(t >> 3);
      const uint64_t at = j < n0 ? j : uint64_t(base) + (j - n0);
      if (at >= S.lcap) continue;
      const uint64_t u = S.list[at];
      if (okey_l(u) != l) continue;
      // the parent's anchor, stepped towards u's side on the lane's axes
      const uint32_t sh = 3u * (D - l + 1);
      const uint64_t m = okey_m(u);
      uint64_t q = (m >> sh) << sh;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if ((t >> a) & 1) {
          const uint64_t unit = 1ull << (sh + a);
          q = ((m >> (sh - 3 + a)) & 1u) ? morton_inc(q, a, unit) : morton_dec(q, a, unit);
        }
      if (q >> (3u * D)) continue;  // outside the domain
      mine[k] = true;
      key[k] = okey(q, l - 1);
      h[k] = set_slot(S, key[k]);
      cur[k] = set_peek(S, h[k]);
    }
#pragma unroll
    for (int k = 0; k < kSetItems; ++k) {
      if (mine[k]) fresh[k] = set_insert(S, key[k], h[k], cur[k]);
      any = any || fresh[k];
    }
    if (__syncthreads_or(any)) set_append(S, fresh, key, wbase, S.count + 2 + (l - 1));
  }
}

// The leaves, in order, from the sorted internal octants: child c of internal
// octant i is internal if its key is in the list, else a leaf.  Its place is
// known from the number a of internal octants that sort before it.  Of the
// octants before a leaf L of level d in the pre-order (a key's ancestors
// before it): an internal one that is not an ancestor of L has all 8 children
// before L; an ancestor has those before the path to L, plus the path's own
// where that is internal.  With S the sum of the path's child numbers that is
// 1 + 8 (a - d) + S + (d - 1) octants, a of them internal: 7 a - 7 d + S leaves.
// (With every ancestor in the list, as the set has for octants inside the
// domain, places lie in [0, 7 nu + 1); no other is written.)
__global__ void balance_leaves(const uint64_t* __restrict__ u, int64_t nu, uint32_t D, uint64_t* __restrict__ out) {
  for (int64_t t = gtid(); t < nu * 8; t += gstride()) {
    const int64_t i = t >> 3;
    const uint64_t k = u[i];
    const uint32_t d = okey_l(k) + 1;
    const uint64_t m = okey_m(k) | (uint64_t(t & 7) << (3u * (D - d)));
    const uint64_t ck = okey(m, d);
    const int64_t a = gallop(u, i + 1, nu, ck);
    if (a < nu && u[a] == ck) continue;
    const int64_t S = __popcll(m & 0x1249249249249249ull) + 2 * __popcll(m & 0x2492492492492492ull) +
                      4 * __popcll(m & 0x4924924924924924ull);
    const int64_t at = 7 * a - 7 * int64_t(d) + S;
    if (at >= 0 && at <= 7 * nu) out[at] = ck;
  }
}

// -------------------------------------------------------------- coarsen --
__device__ __forceinline__ uint32_t child_of(uint64_t ok, uint32_t D) {
  uint32_t l = okey_l(ok);
  if (l == 0) return 0;
  return uint32_t((okey_m(ok) >> (3u * (D - l))) & 7u);
}
// A family (a child-0 leaf followed by its 7 siblings as leaves) becomes its
// parent; other leaves stay.
struct Coarsen {
  const uint64_t* __restrict__ k;
  int64_t n;
  uint32_t D;
  uint64_t* __restrict__ out;
  __device__ bool family(int64_t i) const {
    const uint64_t a = k[i];
    if (i + 7 >= n || okey_l(a) == 0 || child_of(a, D) != 0) return false;
    const uint64_t b = k[i + 7];
    return okey_l(b) == okey_l(a) && parent_key(b, D) == parent_key(a, D);
  }
  __device__ uint32_t count(int64_t i) const {
    for (int d = 1; d <= 7 && i - d >= 0; ++d)
      if (family(i - d)) return 0u;
    return 1u;
  }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    if (c) out[off] = family(i) ? parent_key(k[i], D) : k[i];
  }
};

}  // namespace

static dg_status set_root(dg_octree* out, uint32_t D, cudaStream_t s) {
  out->max_depth = D;
  DG_TRY(out->keys.alloc(1));
  uint64_t root = okey(0, 0);
  DG_CUDA(cudaMemcpyAsync(out->keys.p, &root, 8, cudaMemcpyHostToDevice, s));
  DG_CUDA(cudaStreamSynchronize(s));
  out->n = 1;
  return DG_OK;
}

dg_status points_to_octree(const double* d_pts, int64_t n, uint32_t D, uint32_t m, dg_octree* out, cudaStream_t s) {
  DG_CHECK(D <= kMaxDepth, DG_EDEPTH, "maxDepth above 19 is not supported");
  DG_CHECK(m >= 1, DG_EINVAL, "maxNumPts must be >= 1");
  DG_CHECK(n >= 0, DG_EINVAL, "negative point count");
  if (D == 0 || n <= int64_t(m)) return set_root(out, D, s);  // Construct.C:884-888,915-919
  DBuf<uint64_t> pk, tmp;
  DBuf<uint32_t> sums, cnt;  // cnt: [0] a point outside, [1] leaves with points, [2] leaves
  const int64_t nb = tile_blocks(n + 1);
  DG_TRY(pk.alloc(n));
  DG_TRY(tmp.alloc(n));
  DG_TRY(sums.alloc(nb));
  DG_TRY(cnt.alloc(3));
  DG_CUDA(cudaMemsetAsync(cnt.p, 0, 12, s));
  quantise_points<<<grid_for(n, 256), 256, 0, s>>>(d_pts, n, D, pk.p, cnt.p);
  DG_CUDA(cudaGetLastError());
  DG_TRY(radix_sort_u64(pk, tmp, n, int(3 * D), s));
  // leaf of every point, then adjacent-unique
  point_leaves<<<grid_for(n, 256), 256, 0, s>>>(pk.p, n, D, m, tmp.p);
  DG_CUDA(cudaGetLastError());
  const UniqueKeys uq{tmp.p, pk.p};
  DG_TRY(tile_scan(uq, ItemCount{n}, sums.p, cnt.p + 1, s));
  DG_TRY(tile_emit(uq, ItemCount{n}, sums.p, s));
  // complete the gaps with the coarsest octants
  Gaps gaps{pk.p, cnt.p + 1, D, nullptr};
  const ItemCount ng{n + 1, cnt.p + 1, 1};
  DG_TRY(tile_scan(gaps, ng, sums.p, cnt.p + 2, s));
  uint32_t h[3];
  DG_TRY(read_words(cnt.p, h, 3, s));
  DG_CHECK(!h[0], DG_EINVAL, "points must lie in [0,1)^3");
  DG_TRY(out->keys.alloc(h[2]));
  gaps.out = out->keys.p;
  DG_TRY(tile_emit(gaps, ng, sums.p, s));
  out->n = h[2];
  out->max_depth = D;
  return DG_OK;
}

// Coarsest 2:1 balanced refinement: the set of its internal octants
// (InternalSet), sorted, and the children that are not in it.
dg_status balance_octree(const dg_octree* in, dg_octree* out, cudaStream_t s) {
  const uint32_t D = in->max_depth;
  const int64_t n = in->n;
  DG_CHECK(D <= kMaxDepth, DG_EDEPTH, "maxDepth above 19 is not supported");
  if (n <= 1) {
    out->max_depth = D;
    DG_TRY(out->keys.alloc(n > 0 ? n : 1));
    if (n) DG_CUDA(cudaMemcpyAsync(out->keys.p, in->keys.p, 8 * n, cudaMemcpyDeviceToDevice, s));
    out->n = n;
    return DG_OK;
  }
  constexpr int kCounts = 2 + int(kMaxDepth) + 1;
  DBuf<uint64_t> table, list;
  DBuf<uint32_t> cnt;
  DG_TRY(cnt.alloc(kCounts));
  uint32_t h[kCounts];
  int64_t nu = 0;
  // room for 4 times the internal octants of a complete octree of n leaves
  // (the benchmark's point clouds grow 1.6 to 1.8 times), at most half
  // full; a set that does not fit is built again with four times the room
  for (int64_t lcap = std::max<int64_t>(4096, 4 * (n / 7)); nu == 0; lcap *= 4) {
    DG_CHECK(lcap < (int64_t(1) << 30), DG_ENOMEM, "balance: too many octants");
    const HashShape shape = hash_shape(lcap);
    DG_TRY(table.alloc(int64_t(shape.slots())));
    DG_TRY(list.alloc(lcap));
    DG_CUDA(cudaMemsetAsync(table.p, 0xff, sizeof(uint64_t) * size_t(shape.slots()), s));
    DG_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof h, s));
    const InternalSet S{table.p, shape, list.p, uint32_t(lcap), cnt.p};
    balance_leaf_parents<<<grid_for(n, kSetThreads * kSetItems), kSetThreads, 0, s>>>(in->keys.p, n, D, S);
    for (uint32_t l = D; l-- > 1;) balance_level<<<grid_for(8 * lcap, kSetThreads * kSetItems), kSetThreads, 0, s>>>(l, D, S);
    DG_CUDA(cudaGetLastError());
    DG_TRY(read_words(cnt.p, h, kCounts, s));
    if (h[1]) continue;
    nu = h[0];
    for (int l = 2; l < kCounts; ++l) nu += h[l];
    if (nu == 0) return set_root(out, D, s);
  }
  table.reset();
  DBuf<uint64_t> tmp;
  DG_TRY(tmp.alloc(list.n));
  DG_TRY(radix_sort_u64(list, tmp, nu, int(3 * D + 5), s));
  const int64_t total = 7 * nu + 1;
  DG_CHECK(total < (int64_t(1) << 31), DG_EINVAL, "balance: too many octants");
  DG_TRY(out->keys.alloc(total));
  balance_leaves<<<grid_for(8 * nu, 256), 256, 0, s>>>(list.p, nu, D, out->keys.p);
  DG_CUDA(cudaGetLastError());
  out->n = total;
  out->max_depth = D;
  return DG_OK;
}

dg_status coarsen_octree(const dg_octree* in, dg_octree* out, cudaStream_t s) {
  const uint32_t D = in->max_depth;
  const int64_t n = in->n;
  out->max_depth = D;
  if (n < 8) {  // Coarsen.C:66-70
    DG_TRY(out->keys.alloc(n > 0 ? n : 1));
    if (n) DG_CUDA(cudaMemcpyAsync(out->keys.p, in->keys.p, 8 * n, cudaMemcpyDeviceToDevice, s));
    out->n = n;
    return DG_OK;
  }
  const int64_t nb = tile_blocks(n);
  DBuf<uint32_t> sums;
  DG_TRY(sums.alloc(nb + 1));
  Coarsen f{in->keys.p, n, D, nullptr};
  DG_TRY(tile_scan(f, ItemCount{n}, sums.p, sums.p + nb, s));
  uint32_t total = 0;
  DG_TRY(read_words(sums.p + nb, &total, 1, s));
  DG_TRY(out->keys.alloc(total));
  f.out = out->keys.p;
  DG_TRY(tile_emit(f, ItemCount{n}, sums.p, s));
  out->n = total;
  return DG_OK;
}

}  // namespace dg
