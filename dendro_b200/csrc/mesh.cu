// Mesh (ot::DA) construction on the GPU for one level:
//  * embed the balanced octree at maxDepth+1 and add the positive-boundary
//    pseudo-octants (addBoundaryNodesType1, src/oct/OctFunctions.C:636-716);
//  * flag octants whose anchor is a non-hanging node (flagNodesType3,
//    OctFunctions.C:1501-2025);
//  * number the nodes in DA order (the Vec order of DA::vecGetBuffer,
//    include/oda/oda.txx:948-970) and build the element->node map with
//    hanging masks, child numbers and element types (DA::buildNodeList,
//    src/oda/private/odaBuildNlist.C:47-856; GET_ETYPE_BLOCK,
//    include/oda/odaUtils.h:334).
#include <utility>

#include "octet.cuh"
#include "prim.cuh"

namespace dg {

// (childNum, hanging mask) -> element type in [0,18), 255 when the mask is not
// one of the 18 configurations of include/oda/cnumEtypes.h:19-229.
__constant__ uint8_t c_etype_lut[8][256];

namespace {

// Hanging masks of the 18 element types per child number (cnumEtypes.h).
const uint8_t kEtypeMask[8][18] = {
    {0, 4, 2, 6, 16, 20, 18, 22, 14, 30, 84, 86, 94, 50, 54, 62, 118, 126},
    {0, 1, 8, 9, 32, 33, 40, 41, 13, 45, 49, 57, 61, 168, 169, 173, 185, 189},
    {0, 8, 1, 9, 64, 72, 65, 73, 11, 75, 200, 201, 203, 81, 89, 91, 217, 219},
    {0, 2, 4, 6, 128, 130, 132, 134, 7, 135, 162, 166, 167, 196, 198, 199, 230, 231},
    {0, 1, 32, 33, 64, 65, 96, 97, 35, 99, 69, 101, 103, 224, 225, 227, 229, 231},
    {0, 2, 128, 130, 16, 18, 144, 146, 138, 154, 19, 147, 155, 208, 210, 218, 211, 219},
    {0, 4, 16, 20, 128, 132, 144, 148, 21, 149, 140, 156, 157, 176, 180, 181, 188, 189},
    {0, 8, 64, 72, 32, 40, 96, 104, 76, 108, 42, 106, 110, 112, 120, 124, 122, 126}};

__device__ __forceinline__ int64_t gtid() { return blockIdx.x * int64_t(blockDim.x) + threadIdx.x; }
__device__ __forceinline__ int64_t gstride() { return int64_t(gridDim.x) * blockDim.x; }

__device__ __forceinline__ int64_t find_exact(const uint64_t* __restrict__ a, int64_t n, uint64_t key) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return (lo < n && a[lo] == key) ? lo : -1;
}

// Hash map from the keys of a key array to their places in it: slots of 8
// bytes, a 32-bit tag of the key's hash above the place, so that a table for
// the 672K internal octants of the benchmark mesh (17 MB) stays in L2; a slot
// whose tag matches is checked against the key array, which is sorted or nearly
// so and read with locality.  (Binary searches over the sorted node keys take
// 22 dependent loads each.)
struct KeyMap {
  uint64_t* slot;  // kNoKey: empty
  HashShape shape;
  const uint64_t* keys;
};
__device__ __forceinline__ void map_insert(const KeyMap& M, uint64_t key, uint32_t at) {
  // entries fill at most half the slots, so this ends; tags are below 2^31, so
  // no entry equals the empty slot
  const uint64_t mix = hash_mix(key), wrap = M.shape.slots() - 1;
  const uint64_t e = (uint64_t(hash_tag(mix, M.shape)) << 32) | at;
  uint64_t h = mix >> M.shape.shift;
  while (atomicCAS(reinterpret_cast<unsigned long long*>(M.slot + h), kNoKey, e) != kNoKey) h = (h + 1) & wrap;
}
// The place of `key`, kNoNode when it is not there.
__device__ __forceinline__ uint32_t map_find(const KeyMap& M, uint64_t key) {
  const uint64_t mix = hash_mix(key), wrap = M.shape.slots() - 1;
  const uint32_t tag = hash_tag(mix, M.shape);
  for (uint64_t h = mix >> M.shape.shift;; h = (h + 1) & wrap) {
    const uint64_t cur = M.slot[h];
    if (cur == kNoKey) return kNoNode;
    if (uint32_t(cur >> 32) == tag && M.keys[uint32_t(cur)] == key) return uint32_t(cur);
  }
}

// Per octant its embedded key (level + 1, same anchor) and a byte: bits 0-2
// the positive faces of the domain that it touches, bits 3-7 the number of
// internal octants that it is the first element of.
__global__ void classify_octants(const uint64_t* __restrict__ k, int64_t E, uint32_t D, uint64_t* __restrict__ ekey,
                                 uint8_t* __restrict__ cls) {
  for (int64_t i = gtid(); i < E; i += gstride()) {
    const uint64_t key = k[i];
    ekey[i] = key + 1;
    const uint32_t l = okey_l(key);
    // the coordinates' top l bits are all ones on an axis that touches
    const uint64_t a = okey_m(key) >> (3u * (D - l)), axis = 0x1249249249249249ull & ((1ull << (3u * l)) - 1ull);
    uint32_t f = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) f |= uint32_t(((a >> d) & axis) == axis) << d;
    // its ancestors that do not hold the octant before it: those below the
    // deepest one that holds both (an octree of the root alone: the embedded
    // root, its parent)
    uint32_t c = l ? l : 1u;
    if (i) {
      const uint64_t x = okey_m(key) ^ okey_m(k[i - 1]);
      const uint32_t both = x ? (uint32_t(__clzll(x)) - (64u - 3u * D)) / 3u : D;
      c = l > both + 1 ? l - 1 - both : 0u;
    }
    cls[i] = uint8_t(f | (c << 3));
  }
}

// Per octant its positive-boundary pseudo-octants (embedded keys), one per
// non-empty subset of the faces it touches.
struct PseudoOctants {
  const uint8_t* __restrict__ cls;
  const uint64_t* __restrict__ k;
  uint32_t D;
  uint64_t* __restrict__ out;
  __device__ uint32_t count(int64_t i) const { return (1u << __popc(cls[i] & 7u)) - 1u; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    if (!c) return;
    uint32_t x, y, z;
    demorton(okey_m(k[i]), x, y, z);
    const uint32_t f = cls[i] & 7u, top = 1u << D;
    uint64_t* o = out + off;
    for (uint32_t s = 1; s < 8; ++s)
      if ((s & f) == s)
        *o++ = okey(morton((s & 1) ? top : x, (s & 2) ? top : y, (s & 4) ? top : z), okey_l(k[i]) + 1);
  }
};

// The internal octants (embedded keys), each at its first element, coarser
// first: in key order without a sort; `first` keeps that element.
struct Internals {
  const uint8_t* __restrict__ cls;
  const uint64_t* __restrict__ ekey;
  uint32_t Dp;
  uint64_t* __restrict__ out;
  uint32_t* __restrict__ first;
  __device__ uint32_t count(int64_t i) const { return cls[i] >> 3; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    const uint64_t e = ekey[i];
    for (uint32_t j = 0; j < c; ++j) {
      const uint32_t l = okey_l(e) - c + j;
      out[off + j] = okey(okey_m(e) & ~((1ull << (3u * (Dp - l))) - 1ull), l);
      first[off + j] = uint32_t(i);
    }
  }
};

// Per internal octant: the element ids of its leaf children (kid), its meta
// word, its place in the map of keys, and per child the element anchored at
// the child's anchor (the child, or the first of its own elements; kNoNode in
// an octree with holes).  *covered counts the children, all E elements when no
// octant lies inside another.
__global__ void octet_children(const uint64_t* __restrict__ ukey, const uint32_t* __restrict__ first, int64_t nu,
                               uint32_t Dp, const uint64_t* __restrict__ ekey, int64_t E,
                               uint32_t* __restrict__ umeta, uint32_t* __restrict__ kid,
                               uint32_t* __restrict__ anchored, KeyMap M, uint32_t* __restrict__ covered) {
  uint32_t mine = 0;
  for (int64_t o = gtid(); o < nu; o += gstride()) {
    const uint64_t k = ukey[o], am = okey_m(k);
    const uint32_t m = okey_l(k) + 1;
    const uint32_t sh = 3u * (Dp - m);
    int64_t lo = first[o];
    uint32_t mask = 0;
    // mostly the 8 children are the next 8 elements: read them together
    bool all = lo + 8 <= E;
    if (all) {
      uint64_t e[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) e[c] = ekey[lo + c];
#pragma unroll
      for (int c = 0; c < 8; ++c) all = all && e[c] == okey(am + (uint64_t(c) << sh), m);
    }
    if (all) {
      mask = 255u;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        kid[int64_t(c) * nu + o] = uint32_t(lo + c);
        anchored[int64_t(c) * nu + o] = uint32_t(lo + c);
      }
    } else
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint64_t cm = am + (uint64_t(c) << sh);
      const uint64_t at = lo < E ? ekey[lo] : kNoKey;
      const bool leaf = at == okey(cm, m);
      kid[int64_t(c) * nu + o] = leaf ? uint32_t(lo) : kNoNode;
      anchored[int64_t(c) * nu + o] = lo < E && okey_m(at) == cm ? uint32_t(lo) : kNoNode;
      if (leaf) {
        mask |= 1u << c;
        ++lo;
      } else if (c < 7) {  // refined: past the child's own elements
        lo = gallop(ekey, lo, E, okey(am + (uint64_t(c + 1) << sh), 0));
      }
    }
    umeta[o] = m | (mask << 8);
    map_insert(M, k, uint32_t(o));
    mine += __popc(mask);
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (mine && (threadIdx.x & 31) == 0) atomicAdd(covered, mine);
}

// The octets: the internal octants with leaf children, in order.
struct Octets {
  const uint32_t* __restrict__ umeta;
  const uint32_t* __restrict__ kid;
  int64_t nu, n;
  uint32_t* __restrict__ at;  // [n] the octet's internal octant
  uint32_t* __restrict__ ometa;
  uint32_t* __restrict__ oelem;
  __device__ uint32_t count(int64_t i) const { return ometa_cmask(umeta[i]) ? 1u : 0u; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    if (!c) return;
    at[off] = uint32_t(i);
    ometa[off] = umeta[i];
#pragma unroll
    for (int k = 0; k < 8; ++k) oelem[int64_t(k) * n + off] = kid[int64_t(k) * nu + i];
  }
};

// The place among the internal octants of the parent of octant q (an embedded
// key inside the domain, level >= 1) when q is an element -- when that parent
// has it as a leaf child --, else kNoNode.
__device__ __forceinline__ uint32_t element_parent(const KeyMap& M, const uint32_t* __restrict__ umeta, uint64_t q,
                                                   uint32_t Dp) {
  const uint32_t l = okey_l(q);
  const uint64_t m = okey_m(q);
  const uint32_t o = map_find(M, okey(m & ~((1ull << (3u * (Dp - l + 1))) - 1ull), l - 1));
  return o != kNoNode && ((ometa_cmask(umeta[o]) >> uint32_t((m >> (3u * (Dp - l))) & 7u)) & 1u) ? o : kNoNode;
}
__device__ __forceinline__ bool is_element(const KeyMap& M, const uint32_t* __restrict__ umeta, uint64_t q,
                                           uint32_t Dp) {
  return element_parent(M, umeta, q, Dp) != kNoNode;
}

// NODE flags of the elements (flagNodesType3): the anchor of child c is
// hanging when one of the parent's same-size neighbours across the faces and
// edges of the parent that hold the anchor is an element.  8 lanes per octet:
// lane S looks up the neighbour towards the axes of S, lane c combines them.
__global__ void flag_elements(const uint64_t* __restrict__ okeys, int64_t n, uint32_t Dp,
                              const uint32_t* __restrict__ ometa, const uint32_t* __restrict__ oelem, KeyMap M,
                              uint8_t* __restrict__ flag) {
  const int64_t nr = (8 * n + 31) & ~int64_t(31);
  for (int64_t t = gtid(); t < nr; t += gstride()) {
    const int64_t o = t >> 3;
    const uint32_t c = uint32_t(t & 7);
    bool coarse = false;
    uint32_t e = kNoNode;
    if (o < n) {
      e = oelem[int64_t(c) * n + o];
      const uint64_t k = okeys[o];
      const uint32_t pl = okey_l(k);
      if (pl >= 1 && c != 0 && c != 7) {
        const uint64_t unit = 1ull << (3u * (Dp - pl));
        uint64_t q = okey_m(k);
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if ((c >> a) & 1) q = morton_dec(q, a, unit << a);
        if (!(q >> (3u * Dp))) coarse = is_element(M, ometa, okey(q, pl), Dp);
      }
    }
    const uint32_t L = __ballot_sync(0xffffffffu, coarse) >> (threadIdx.x & 24);
    if (e == kNoNode) continue;
    bool hanging = false;
    if (c != 0 && c != 7)
#pragma unroll
      for (uint32_t S = 1; S < 7; ++S) hanging = hanging || (!(S & c) && ((L >> S) & 1u));
    flag[e] = hanging ? 0 : 1;
  }
}

// The same for the pseudo-octants (their neighbours may be pseudo-octants).
__global__ void flag_pseudo(const uint64_t* __restrict__ ps, int64_t P, uint32_t Dp,
                            const uint32_t* __restrict__ ometa, KeyMap M, uint8_t* __restrict__ flag) {
  const uint64_t outside = okey(1ull << (3u * (Dp - 1)), 0);
  for (int64_t i = gtid(); i < P; i += gstride()) {
    const uint64_t k = ps[i];
    const uint32_t m = okey_l(k);
    bool hanging = false;
    if (m > 1) {
      uint32_t x, y, z;
      demorton(okey_m(k), x, y, z);
      const uint32_t s = 1u << (Dp - m);
      const uint32_t c = uint32_t((okey_m(k) >> (3u * (Dp - m))) & 7u);
      if (c != 0 && c != 7) {
        const uint32_t zero = (~c) & 7u, pmask = ~((2u * s) - 1u);
        for (uint32_t S = 1; S < 8 && !hanging; ++S) {
          if ((S & zero) != S) continue;
          if (((S & 1) && !x) || ((S & 2) && !y) || ((S & 4) && !z)) continue;
          const uint32_t nx = x - ((S & 1) ? s : 0), ny = y - ((S & 2) ? s : 0), nz = z - ((S & 4) ? s : 0);
          const uint64_t q = okey(morton(nx & pmask, ny & pmask, nz & pmask), m - 1);
          hanging = q >= outside ? find_exact(ps, P, q) >= 0 : is_element(M, ometa, q, Dp);
        }
      }
    }
    flag[i] = hanging ? 0 : 1;
  }
}

// The nodes: octants flagged NODE, elements then pseudo-octants, in key
// order (pseudo-octants lie outside the domain child of the embedded root, so
// they sort after every element); rank[i] = the node id of octant i's anchor.
struct NodeKeys {
  const uint8_t* __restrict__ flag;
  const uint64_t* __restrict__ ekey;
  int64_t E;
  const uint64_t* __restrict__ ps;
  uint64_t* __restrict__ nkey;
  uint32_t* __restrict__ rank;
  __device__ uint32_t count(int64_t i) const { return flag[i]; }
  __device__ void emit(int64_t i, uint32_t off, uint32_t c) const {
    rank[i] = c ? off : kNoNode;
    if (c) nkey[off] = okey_m(i < E ? ekey[i] : ps[i - E]);
  }
};

// The node ids of the anchors of an internal octant's 8 children, 32 bytes each.
__global__ void octet_own_nodes(int64_t nu, const uint32_t* __restrict__ anchored, const uint32_t* __restrict__ rank,
                                uint32_t* __restrict__ own) {
  for (int64_t o = gtid(); o < nu; o += gstride()) {
    uint32_t v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t e = anchored[int64_t(c) * nu + o];
      v[c] = e != kNoNode ? rank[e] : kNoNode;
    }
    reinterpret_cast<uint4*>(own)[2 * o] = make_uint4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<uint4*>(own)[2 * o + 1] = make_uint4(v[4], v[5], v[6], v[7]);
  }
}

// Children of an octet that have lattice point p as a vertex.
__host__ __device__ constexpr uint32_t lat_children(int p) {
  uint32_t t = 0;
  for (int c = 0; c < 8; ++c) {
    bool in = true;
    for (int a = 0; a < 3; ++a) {
      const int d = oct_coord(p, a) - ((c >> a) & 1);
      in = in && (d == 0 || d == 1);
    }
    if (in) t |= 1u << c;
  }
  return t;
}
// Corners of the octet that a hanging point p interpolates from.
__host__ __device__ constexpr uint32_t lat_corners(int p) {
  uint32_t t = 0;
  for (int v = 0; v < 8; ++v) {
    bool in = true;
    for (int a = 0; a < 3; ++a) in = in && (oct_coord(p, a) == 1 || oct_coord(p, a) == 2 * ((v >> a) & 1));
    if (in) t |= 1u << (2 * (v & 1) + 6 * ((v >> 1) & 1) + 18 * ((v >> 2) & 1));
  }
  return t;
}
struct LatticeTables {
  uint32_t children[32], corners[32];
  constexpr LatticeTables() : children(), corners() {
    for (int p = 0; p < 27; ++p) {
      children[p] = lat_children(p);
      corners[p] = lat_corners(p);
    }
  }
};
__constant__ LatticeTables c_lat = LatticeTables();

// The node at point m outside the domain: a pseudo-octant's anchor or none.
struct PseudoNodes {
  const uint64_t* __restrict__ ps;
  int64_t P;
  const uint32_t* __restrict__ rank;  // node ids of the pseudo-octants
  __device__ uint32_t operator()(uint64_t m) const {
    const int64_t i = gallop(ps, 0, P, okey(m, 0));
    return i < P && okey_m(ps[i]) == m ? rank[i] : kNoNode;
  }
};

// Element -> node map, hanging masks, element types and the octets' lattice
// ids.  An octet's lattice points with coordinates 0 and 1 are its children's
// anchors; one with a coordinate 2 on the axes of S is a child's anchor of the
// neighbour cell of the parent's size towards S, so 7 look-ups among the
// internal octants give all 27 points (a look-up per point in a hash of the
// nodes took 553 us on the 4.7M-element benchmark mesh, and 248 us to fill).  A
// neighbour that is not internal is an element, which has a node at most at
// its anchor, or lies inside an element of twice the size, with a node at most
// where their anchors meet; both are found through their parents.  A vertex
// without a node hangs and lists its parent's vertex, an octet corner
// (DA::buildNodeList).  8 lanes per octet, lane S for the neighbour towards S
// (0: the octet itself); a CTA works 32 octets and writes their rows together.
constexpr int kLatOctets = 32;
__global__ void __launch_bounds__(256) octet_lattice(const uint64_t* __restrict__ ukey,
                                                     const uint32_t* __restrict__ umeta,
                                                     const uint32_t* __restrict__ own, KeyMap M,
                                                     const uint32_t* __restrict__ oat, int64_t n, uint32_t Dp,
                                                     const uint32_t* __restrict__ ometa,
                                                     const uint32_t* __restrict__ oelem, PseudoNodes F, int64_t E,
                                                     uint32_t* __restrict__ oid, uint32_t* __restrict__ nl,
                                                     uint32_t* __restrict__ meta, uint32_t* __restrict__ err) {
  __shared__ uint32_t sid[27][kLatOctets + 1], shang[kLatOctets];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint64_t outside = 1ull << (3u * (Dp - 1));
  constexpr int kPer = kLatOctets / 8;  // octets per warp
  const uint32_t touch = lane < 27 ? c_lat.children[lane] : 0u, corner = lane < 27 ? c_lat.corners[lane] : 0u;
  constexpr uint32_t kNever = (1u << 0) | (1u << 2) | (1u << 6) | (1u << 8) | (1u << 13) | (1u << 18) | (1u << 20) |
                              (1u << 24) | (1u << 26);  // corners and the centre do not hang
  for (int64_t o0 = int64_t(blockIdx.x) * kLatOctets; o0 < n; o0 += int64_t(gridDim.x) * kLatOctets) {
    {
      const int j = tid >> 3;
      const uint32_t S = tid & 7;
      const int64_t o = o0 + j;
      if (o < n) {
        uint32_t q = oat[o];
        const uint64_t k = ukey[q];
        const uint32_t pl = okey_l(k);
        uint64_t am = okey_m(k);
        if (S) {
          const uint64_t unit = 1ull << (3u * (Dp - pl));
#pragma unroll
          for (int a = 0; a < 3; ++a)
            if ((S >> a) & 1) am = morton_inc(am, a, unit << a);
          q = am < outside ? map_find(M, okey(am, pl)) : kNoNode;
        }
        const uint32_t sh = 3u * (Dp - pl - 1);
        uint32_t v[8];
        if (am >= outside || pl == 0) {
          // (the root octant alone: its octet's other children are outside)
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint64_t m = am + (uint64_t(c) << sh);
            v[c] = uint32_t(c) & S ? kNoNode : m >= outside ? F(m) : own[8 * int64_t(q) + c];
          }
        } else if (q != kNoNode) {
          const uint4 a = reinterpret_cast<const uint4*>(own)[2 * int64_t(q)];
          const uint4 b = reinterpret_cast<const uint4*>(own)[2 * int64_t(q) + 1];
          v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
          v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) v[c] = kNoNode;
          // the cell an element, or the first child's place in one (or more
          // than one) size up
          for (uint32_t l = pl; l >= 1; --l) {
            const uint32_t child = uint32_t((am >> (3u * (Dp - l))) & 7u);
            const uint32_t par = element_parent(M, umeta, okey(am, l), Dp);
            if (par != kNoNode) {
              v[0] = own[8 * int64_t(par) + child];
              break;
            }
            if (child) break;
          }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (!(uint32_t(c) & S)) {
            // per axis: 2 where S, else the child's bit
            const int px = (S & 1) ? 2 : (c & 1), py = (S & 2) ? 2 : ((c >> 1) & 1), pz = (S & 4) ? 2 : (c >> 2);
            sid[px + 3 * py + 9 * pz][j] = v[c];
          }
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int j = w * kPer + i;
      const int64_t o = o0 + j;
      if (o >= n) break;  // the same for the whole warp
      const uint32_t id = lane < 27 ? sid[lane][j] : kNoNode;
      const bool present = (ometa_cmask(ometa[o]) & touch) != 0u, found = id != kNoNode;
      const uint32_t hang = __ballot_sync(0xffffffffu, present && !found);
      const uint32_t need = __reduce_or_sync(0xffffffffu, ((hang >> lane) & 1u) ? corner : 0u);
      if (((need >> lane) & 1u) && !found) atomicOr(err, 1u);
      if (lane < 27 && !present && !((need >> lane) & 1u)) sid[lane][j] = kNoNode;
      if (lane == 0) {
        shang[j] = hang;
        if (hang & kNever) atomicOr(err, 2u);
      }
    }
    __syncthreads();
    for (int i = tid; i < 27 * kLatOctets; i += 256) {
      const int p = i / kLatOctets, j = i % kLatOctets;
      if (o0 + j < n) oid[int64_t(p) * n + o0 + j] = sid[p][j];
    }
    {
      const int j = tid >> 3, c = tid & 7;
      const int64_t o = o0 + j;
      const uint32_t e = o < n ? oelem[int64_t(c) * n + o] : kNoNode;
      if (e != kNoNode) {
        const uint32_t hang = shang[j];
        uint32_t mask = 0;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          int p = ((c & 1) + (v & 1)) + 3 * (((c >> 1) & 1) + ((v >> 1) & 1)) + 9 * ((c >> 2) + (v >> 2));
          if ((hang >> p) & 1u) {
            mask |= 1u << v;
            p = 2 * (v & 1) + 6 * ((v >> 1) & 1) + 18 * (v >> 2);
          }
          nl[int64_t(v) * E + e] = sid[p][j];
        }
        uint32_t t = mask ? c_etype_lut[c][mask] : 0u;
        if (t == 255u) {
          atomicOr(err, 2u);
          t = 0;
        }
        meta[e] = meta_pack(ometa_lev(ometa[o]), uint32_t(c), mask, t);
      }
    }
    __syncthreads();
  }
}

// Exclusive scan of one value per thread over a block of TE threads (every
// thread calls it); the block total is returned through `total`.
template <int TE>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* wsum, uint32_t& total) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  uint32_t base = 0;
  total = 0;
  for (int i = 0; i < TE / 32; ++i) {
    if (i < w) base += wsum[i];
    total += wsum[i];
  }
  __syncthreads();
  return base + incl - v;
}

// Per tile of TE consecutive elements (one CTA of TE threads per tile): the
// 8 TE (node id, position v * TE + element) pairs are sorted in shared memory
// by a bitonic network; the sorted positions are the tile's references
// grouped by node (inc), the distinct ids its node list (to tmp, count to
// cnt) and the run ends per node nend.
template <int TE>
__global__ void __launch_bounds__(TE) tile_lists(const uint32_t* __restrict__ nl, int64_t E, int64_t ntiles,
                                                 uint32_t* __restrict__ tmp, uint32_t* __restrict__ cnt,
                                                 uint16_t* __restrict__ nend, uint16_t* __restrict__ inc,
                                                 uint8_t* __restrict__ eloc8) {
  constexpr int S = 8 * TE;
  constexpr int kPer = 8;  // sorted entries per thread
  static_assert(S <= 4096, "positions are 12-bit");
  extern __shared__ __align__(16) unsigned char tl_smem[];
  uint64_t* key = reinterpret_cast<uint64_t*>(tl_smem);
  uint16_t* slot = reinterpret_cast<uint16_t*>(key + S);  // position -> node rank
  __shared__ uint32_t wsum[TE / 32];
  const int tid = threadIdx.x;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    for (int i = tid; i < S; i += TE) {
      const int v = i / TE, el = i % TE;
      const int64_t e = t * TE + el;
      key[i] = e < E ? (uint64_t(nl[int64_t(v) * E + e]) << 12) | uint64_t(i) : ~0ull;
    }
    __syncthreads();
    for (int k = 2; k <= S; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int p = tid; p < S / 2; p += TE) {
          const int i = 2 * p - (p & (j - 1));  // lower index of the pair, bit j clear
          const int l = i + j;
          const bool up = (i & k) == 0;
          const uint64_t a = key[i], b = key[l];
          if ((a > b) == up) {
            key[i] = b;
            key[l] = a;
          }
        }
        __syncthreads();
      }
    uint32_t first_f = 0, nfirst = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int j = tid * kPer + q;
      const uint64_t kj = key[j];
      const bool first = kj != ~0ull && (j == 0 || (key[j - 1] >> 12) != (kj >> 12));
      first_f |= uint32_t(first) << q;
      nfirst += first;
    }
    uint32_t total = 0;
    uint32_t run = block_excl_scan<TE>(nfirst, wsum, total);
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int j = tid * kPer + q;
      const uint64_t kj = key[j];
      if (kj == ~0ull) continue;
      if ((first_f >> q) & 1u) {
        tmp[t * S + run] = uint32_t(kj >> 12);
        ++run;
      }
      inc[t * S + j] = uint16_t(kj & 4095u);
      slot[kj & 4095u] = uint16_t(run - 1);
      const bool last = j + 1 == S || (key[j + 1] >> 12) != (kj >> 12);  // padding keys end every run
      if (last) nend[t * S + run - 1] = uint16_t(j + 1);
    }
    if (tid == 0) cnt[t] = total;
    __syncthreads();
    {  // per element the node ranks of its eight vertices (at most 256 nodes)
      const int64_t e = t * TE + tid;
      if (e < E) {
        uint2 o;
        o.x = uint32_t(slot[0 * TE + tid]) | (uint32_t(slot[1 * TE + tid]) << 8) |
              (uint32_t(slot[2 * TE + tid]) << 16) | (uint32_t(slot[3 * TE + tid]) << 24);
        o.y = uint32_t(slot[4 * TE + tid]) | (uint32_t(slot[5 * TE + tid]) << 8) |
              (uint32_t(slot[6 * TE + tid]) << 16) | (uint32_t(slot[7 * TE + tid]) << 24);
        reinterpret_cast<uint2*>(eloc8)[e] = o;
      }
      __syncthreads();
    }
  }
}

// Copy each tile's node list (capacity S per tile) to its final place.
__global__ void tile_compact(const uint32_t* __restrict__ tmp, int S, const uint32_t* __restrict__ ptr,
                             int64_t ntiles, uint32_t* __restrict__ out) {
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint32_t p0 = ptr[t], n = ptr[t + 1] - p0;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) out[p0 + k] = tmp[t * S + k];
  }
}

// Warp-tile reference lists in bytes, per tile of kWarpTile elements (768
// bytes): the 8 * kWarpTile references sorted by node as positions
// v * kWarpTile + element, the node's rank in the tile list, and flags for
// the kernel's segmented sum, which gives each lane 8 consecutive references:
// 1 = a new sum starts here, 2 = the sum leaves after this reference, 4 = it
// leaves as a store (the node's whole run lies in this lane and no other
// tile uses the node), 8 = valid reference.  One warp per tile, one lane per
// node; runs after the nodes shared between tiles are marked.
__global__ void warp_refs(const uint16_t* __restrict__ inc, const uint16_t* __restrict__ nend,
                          const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ nodes,
                          const uint32_t* __restrict__ meta, int64_t ntiles, uint8_t* __restrict__ tmp,
                          uint8_t* __restrict__ out) {
  constexpr int S = 8 * kWarpTile;
  const int lane = threadIdx.x & 31;
  const int64_t nw = int64_t(gridDim.x) * (blockDim.x / 32);
  for (int64_t t = blockIdx.x * int64_t(blockDim.x / 32) + (threadIdx.x >> 5); t < ntiles; t += nw) {
    uint8_t* o = tmp + t * 3 * S;  // positions, ranks, flag bytes (8 valid, 1 start, 2 leave, 4 store)
    for (int j = lane; j < S; j += 32) o[2 * S + j] = 0;  // invalid until written
    __syncwarp();
    const uint32_t p0 = ptr[t], nt = ptr[t + 1] - p0;
    for (uint32_t k = lane; k < nt; k += 32) {
      const uint32_t beg = k ? nend[t * S + k - 1] : 0u, end = nend[t * S + k];
      const bool excl = !(nodes[p0 + k] & 0x80000000u);
      for (uint32_t j = beg; j < end; ++j) {
        o[j] = uint8_t(inc[t * S + j]);
        o[S + j] = uint8_t(k);
        const bool lane_first = (j & 7u) == 0u, lane_last = (j & 7u) == 7u;
        const bool start = j == beg || lane_first;
        const bool flush = j + 1 == end || lane_last;
        const bool whole = (beg >> 3) == ((end - 1) >> 3);  // the run does not cross a lane boundary
        o[2 * S + j] = uint8_t(8u | (start ? 1u : 0u) | (flush ? 2u : 0u) | (flush && whole && excl ? 4u : 0u));
      }
    }
    __syncwarp();
    // per lane its 8 references: positions v * 32 + element become frame
    // positions (v ^ c) * 32 + element, the flag bytes one word of bit masks
    uint8_t* f = out + t * kWarpRefBytes;
    uint32_t word = 0;
    for (int q = 0; q < 8; ++q) {
      const int j = lane * 8 + q;
      const uint32_t fl = o[2 * S + j];
      uint32_t pf = 0, rk = 0;
      if (fl & 8u) {
        const uint32_t pos = o[j];
        const uint32_t c = meta_cnum(meta[t * kWarpTile + (pos & 31u)]);
        pf = (((pos >> 5) ^ c) << 5) | (pos & 31u);
        rk = o[S + j];
        word |= (1u << q) | ((fl & 1u) << (8 + q)) | (((fl >> 1) & 1u) << (16 + q)) | (((fl >> 2) & 1u) << (24 + q));
      }
      f[j] = uint8_t(pf);
      f[S + j] = uint8_t(rk);
    }
    reinterpret_cast<uint32_t*>(f + 2 * S)[lane] = word;
    __syncwarp();
  }
}

// Warp tiles: node ranks in the child-number frame and the per-element word
// (level, frame hanging mask).
__global__ void warp_frame(const uint32_t* __restrict__ meta, int64_t E, uint2* __restrict__ eloc8,
                           uint32_t* __restrict__ wmeta) {
  for (int64_t e = gtid(); e < E; e += gstride()) {
    const uint32_t m = meta[e];
    eloc8[e] = xor_perm_bytes(eloc8[e], meta_cnum(m));
    wmeta[e] = wmeta_pack(m);
  }
}

// Per node, the number of tiles whose list holds it.
// An entry whose bit 31 is already set (a warp-tile node whose references
// span two lanes of the segmented sum) counts twice, so that it is treated
// like a node shared between tiles.
__global__ void tile_touch(const uint32_t* __restrict__ nodes, int64_t n, uint32_t* __restrict__ touch) {
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const uint32_t id = nodes[i];
    atomicAdd(touch + (id & 0x7fffffffu), (id & 0x80000000u) ? 2u : 1u);
  }
}

// Warp tiles: mark (bit 31) the nodes whose run of sorted references crosses
// a boundary between two lanes' groups of 8, since their sums arrive in parts.
__global__ void warp_split_runs(const uint16_t* __restrict__ nend, const uint32_t* __restrict__ ptr, int64_t ntiles,
                                uint32_t* __restrict__ nodes) {
  constexpr int S = 8 * kWarpTile;
  const int lane = threadIdx.x & 31;
  const int64_t nw = int64_t(gridDim.x) * (blockDim.x / 32);
  for (int64_t t = blockIdx.x * int64_t(blockDim.x / 32) + (threadIdx.x >> 5); t < ntiles; t += nw) {
    const uint32_t p0 = ptr[t], nt = ptr[t + 1] - p0;
    for (uint32_t k = lane; k < nt; k += 32) {
      const uint32_t beg = k ? nend[t * S + k - 1] : 0u, end = nend[t * S + k];
      if ((beg >> 3) != ((end - 1) >> 3)) nodes[p0 + k] |= 0x80000000u;
    }
  }
}

// Bit 31 of a list entry: the node is referenced by more than one tile, so its
// sum must be accumulated with a global atomic.
__global__ void tile_local_mark(uint32_t* __restrict__ nodes, int64_t n, const uint32_t* __restrict__ touch) {
  for (int64_t i = gtid(); i < n; i += gstride()) {
    const uint32_t id = nodes[i] & 0x7fffffffu;
    if (touch[id] > 1u) nodes[i] = id | 0x80000000u;
  }
}

}  // namespace

static dg_status upload_etype_lut() {
  static bool done = false;
  if (done) return DG_OK;
  uint8_t lut[8][256];
  memset(lut, 255, sizeof lut);
  for (int c = 0; c < 8; ++c)
    for (int t = 0; t < 18; ++t) lut[c][kEtypeMask[c][t]] = uint8_t(t);
  DG_CUDA(cudaMemcpyToSymbol(c_etype_lut, lut, sizeof lut));
  DG_CUDA(cudaStreamSynchronize(nullptr));  // there before kernels on other streams
  done = true;
  return DG_OK;
}

dg_status build_mesh(const dg_octree* tree, dg_da* da, cudaStream_t s) {
  const uint32_t D = tree->max_depth;
  const int64_t E = tree->n;
  DG_CHECK(D + 1 <= kMaxEmbeddedDepth, DG_EDEPTH,
           "mesh: maxDepth above 18 is not supported (the embedded depth's keys would exceed 64 bits)");
  DG_CHECK(E >= 1, DG_EINVAL, "empty octree");
  DG_TRY(upload_etype_lut());
  DG_CHECK(E < (int64_t(1) << 31), DG_EINVAL, "mesh above 2^31 elements");
  const uint32_t Dp = D + 1;
  OctetSet& O = da->octs;
  da->D = Dp;
  da->E = E;
  DG_TRY(da->ekey.alloc(E));
  const int64_t nb = tile_blocks(E);
  DBuf<uint32_t> sums, cnt;  // cnt: [0] pseudo-octants, [1] internal octants, [2] nodes, [3] children, [4] errors, [5] octets
  DG_TRY(sums.alloc(2 * nb));
  DG_TRY(cnt.alloc(6));
  DG_CUDA(cudaMemsetAsync(cnt.p, 0, 24, s));
  DBuf<uint8_t> cls;
  DG_TRY(cls.alloc(E));
  classify_octants<<<grid_for(E, 256), 256, 0, s>>>(tree->keys.p, E, D, da->ekey.p, cls.p);
  PseudoOctants pf{cls.p, tree->keys.p, D, nullptr};
  Internals uf{cls.p, da->ekey.p, Dp, nullptr, nullptr};
  DG_TRY(tile_scan(pf, ItemCount{E}, sums.p, cnt.p, s));
  DG_TRY(tile_scan(uf, ItemCount{E}, sums.p + nb, cnt.p + 1, s));
  uint32_t h[6];
  DG_TRY(read_words(cnt.p, h, 2, s));
  const int64_t P = h[0], nu = h[1];
  da->P = P;
  DBuf<uint64_t> ps, pt, ukey;
  DBuf<uint32_t> first;
  DG_TRY(ps.alloc(P));
  DG_TRY(pt.alloc(P));
  DG_TRY(ukey.alloc(nu));
  DG_TRY(first.alloc(nu));
  pf.out = ps.p;
  uf.out = ukey.p;
  uf.first = first.p;
  DG_TRY(tile_emit(pf, ItemCount{E}, sums.p, s));
  DG_TRY(tile_emit(uf, ItemCount{E}, sums.p + nb, s));
  // Pseudo-octants are made in the order of their octants.  The octants that
  // touch a face of the domain are, in their order, ordered on that face (and
  // so for edges), so the pseudo-octants beyond one face, edge or corner are
  // sorted already, and those 7 kinds sort by the top bits of the coordinates:
  // one stable pass on 3 bits sorts them all.
  DG_TRY(radix_sort_u64(ps, pt, P, 3, s, int(5 + 3 * D)));
  DBuf<uint64_t> slots;
  DBuf<uint32_t> anchored, kid, umeta;
  DG_TRY(anchored.alloc(8 * nu));
  DG_TRY(kid.alloc(8 * nu));
  DG_TRY(umeta.alloc(nu));
  const HashShape shape = hash_shape(nu);
  DG_TRY(slots.alloc(int64_t(shape.slots())));
  DG_CUDA(cudaMemsetAsync(slots.p, 0xff, sizeof(uint64_t) * size_t(slots.n), s));
  const KeyMap um{slots.p, shape, ukey.p};
  octet_children<<<grid_for(nu, 128, 16), 128, 0, s>>>(ukey.p, first.p, nu, Dp, da->ekey.p, E, umeta.p, kid.p, anchored.p,
                                                   um, cnt.p + 3);
  DBuf<uint8_t> flag;
  DG_TRY(flag.alloc(E + P));
  flag_elements<<<grid_for(8 * nu, 256), 256, 0, s>>>(ukey.p, nu, Dp, umeta.p, kid.p, um, flag.p);
  if (P) flag_pseudo<<<grid_for(P, 128), 128, 0, s>>>(ps.p, P, Dp, umeta.p, um, flag.p + E);
  DG_CUDA(cudaGetLastError());
  NodeKeys nf{flag.p, da->ekey.p, E, ps.p, nullptr, nullptr};
  Octets of{umeta.p, kid.p, nu, 0, nullptr, nullptr, nullptr};
  DBuf<uint32_t> nsums, rank, own, oat;
  const int64_t nbn = tile_blocks(E + P);
  DG_TRY(nsums.alloc(nbn + tile_blocks(nu)));
  DG_TRY(tile_scan(nf, ItemCount{E + P}, nsums.p, cnt.p + 2, s));
  DG_TRY(tile_scan(of, ItemCount{nu}, nsums.p + nbn, cnt.p + 5, s));
  DG_TRY(read_words(cnt.p, h, 6, s));
  DG_CHECK(h[3] == uint32_t(E), DG_EUNBALANCED, "octants inside one another: octree not linear");
  const int64_t N = h[2], n = h[5];
  da->N = N;
  DG_TRY(da->nkey.alloc(N));
  DG_TRY(rank.alloc(E + P));
  DG_TRY(own.alloc(8 * nu));
  nf.nkey = da->nkey.p;
  nf.rank = rank.p;
  DG_TRY(tile_emit(nf, ItemCount{E + P}, nsums.p, s));
  octet_own_nodes<<<grid_for(nu, 256), 256, 0, s>>>(nu, anchored.p, rank.p, own.p);
  DG_TRY(oat.alloc(n));
  DG_TRY(O.meta.alloc(n));
  DG_TRY(O.elem.alloc(8 * n));
  DG_TRY(O.id.alloc(27 * n));
  DG_TRY(da->nl.alloc(8 * E));
  DG_TRY(da->meta.alloc(E));
  of.n = n;
  of.at = oat.p;
  of.ometa = O.meta.p;
  of.oelem = O.elem.p;
  DG_TRY(tile_emit(of, ItemCount{nu}, nsums.p + nbn, s));
  const PseudoNodes pn{ps.p, P, rank.p + E};
  octet_lattice<<<grid_for(n, kLatOctets, 8), 256, 0, s>>>(ukey.p, umeta.p, own.p, um, oat.p, n, Dp, O.meta.p,
                                                           O.elem.p, pn, E, O.id.p, da->nl.p, da->meta.p, cnt.p + 4);
  DG_CUDA(cudaGetLastError());
  DG_TRY(read_words(cnt.p, h, 5, s));
  DG_CHECK(!(h[4] & 1u), DG_EUNBALANCED, "hanging vertex without a parent node: octree not 2:1 balanced");
  DG_CHECK(!(h[4] & 2u), DG_EUNBALANCED, "hanging configuration outside the 18 element types");
  O.n = n;
  return DG_OK;
}

template <int TE>
static dg_status launch_tile_lists(const dg_da* da, int64_t nt, uint32_t* tmp, uint32_t* cnt, uint16_t* nend,
                                   uint16_t* inc, uint8_t* eloc8, cudaStream_t s) {
  const size_t smem = size_t(8 + 2) * 8 * TE;
  static bool set = false;
  if (!set && smem > 48 * 1024) {
    DG_CUDA(cudaFuncSetAttribute(tile_lists<TE>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  }
  set = true;
  tile_lists<TE><<<grid_for(nt, TE, 2048 / TE), TE, smem, s>>>(da->nl.p, da->E, nt, tmp, cnt, nend, inc, eloc8);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}

// One wait, for the length of the node lists: the first application on a mesh
// has this before it.
static dg_status build_tile_set(const dg_da* da, TileSet& ts, cudaStream_t s) {
  DG_CHECK(da->N < (int64_t(1) << 31), DG_EINVAL, "mesh above 2^31 nodes");
  constexpr int S = 8 * kWarpTile;
  const int64_t E = da->E, nt = (E + kWarpTile - 1) / kWarpTile;
  DBuf<uint32_t> tmp, cnt, touch;
  DBuf<uint16_t> nend, inc;  // tile t, node k -> end of its run in inc, the references ordered by node
  DBuf<uint8_t> r3;
  DG_TRY(tmp.alloc(nt * S));
  DG_TRY(cnt.alloc(nt + 1));
  DG_TRY(nend.alloc(nt * S));
  DG_TRY(inc.alloc(nt * S));
  DG_TRY(ts.eloc8.alloc(8 * nt * kWarpTile));  // whole tiles
  DG_CUDA(cudaMemsetAsync(cnt.p + nt, 0, 4, s));
  DG_TRY(launch_tile_lists<kWarpTile>(da, nt, tmp.p, cnt.p, nend.p, inc.p, ts.eloc8.p, s));
  DG_TRY(ts.ptr.alloc(nt + 1));
  DG_TRY(scan_u32(cnt.p, ts.ptr.p, nt + 1, nullptr, s));
  uint32_t total = 0;
  DG_TRY(read_words(ts.ptr.p + nt, &total, 1, s));
  DG_TRY(ts.nodes.alloc(total + kNodePad));
  tile_compact<<<grid_for(nt, 256, 8), 256, 0, s>>>(tmp.p, S, ts.ptr.p, nt, ts.nodes.p);
  DG_TRY(touch.alloc(da->N));
  DG_CUDA(cudaMemsetAsync(touch.p, 0, 4 * da->N, s));
  warp_split_runs<<<grid_for(nt * 32, 256, 8), 256, 0, s>>>(nend.p, ts.ptr.p, nt, ts.nodes.p);
  tile_touch<<<grid_for(total, 256), 256, 0, s>>>(ts.nodes.p, total, touch.p);
  tile_local_mark<<<grid_for(total, 256), 256, 0, s>>>(ts.nodes.p, total, touch.p);
  DG_TRY(r3.alloc(nt * 3 * S));
  DG_TRY(ts.ref8.alloc(nt * kWarpRefBytes));
  warp_refs<<<grid_for(nt * 32, 256, 8), 256, 0, s>>>(inc.p, nend.p, ts.ptr.p, ts.nodes.p, da->meta.p, nt, r3.p,
                                                       ts.ref8.p);
  DG_TRY(ts.wmeta.alloc(nt * kWarpTile));  // whole tiles
  warp_frame<<<grid_for(E, 256), 256, 0, s>>>(da->meta.p, E, reinterpret_cast<uint2*>(ts.eloc8.p), ts.wmeta.p);
  DG_CUDA(cudaGetLastError());
  ts.ntiles = nt;
  return DG_OK;
}

dg_status ensure_tiles(dg_da* da, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(da->tables);
  if (da->tiles_ready) return DG_OK;
  DG_TRY(build_table(
      s, [&](cudaStream_t t) { return build_tile_set(da, da->tiles_w, t); },
      [&] { da->tiles_w = TileSet(); }));
  da->tiles_ready = true;
  return DG_OK;
}

uint32_t etype_mask(int c, int t) { return kEtypeMask[c & 7][t % 18]; }

}  // namespace dg
