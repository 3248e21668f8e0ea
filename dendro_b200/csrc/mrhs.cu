// Multi-right-hand-side operator Y = A X: the scalar Laplacian + mass operator
// (JAC_TYPE2_ELEM_MULT_BLOCK, examples/src/backend/omgNeumann.C:468-488) applied
// to nrhs vectors at once, X and Y node-major [N][nrhs].  The reference applies
// MatMult to one vector at a time; the batching has no reference counterpart.
//
// The octet kernels below run on the CUDA cores with exact products in the
// vectors' precision; mrhs_tc.cu has the contraction on the 5th-generation
// tensor cores.  (Contractions per element on mma.sync, TF32 in one or three
// products, took 2120 and 2231 us for 64 right-hand sides on the 2.9M-element
// benchmark mesh, bound by L1, where the pair kernel takes 1140 us.)
#include <algorithm>

#include "octet.cuh"

namespace dg {

namespace {

constexpr int kRC = 16;  // right-hand sides come in multiples of this

// FP64: a group of G lanes (32, or 16 for the last 16 right-hand sides) per octet
// and G right-hand sides, one lane per right-hand side.  Each lane holds its
// column's 27 lattice values of the octet in registers and runs the octet
// arithmetic of the scalar kernel (octet_apply: hanging points, the children's
// Walsh-form element operators, T^T); the octet's node ids, meta word and
// element ids are the same for the whole group, and the X rows read and the Y
// rows added are G consecutive values per node.  Each group copies those 36
// words of the task one grid stride ahead into its own shared-memory slot
// (4-byte cp.async) while it works the current task, so the X row loads of a
// task issue without the round trip for its ids.  Y must be zero on entry (the
// sums leave with global reductions; the centre of a full octet with a store).
// Works the nb blocks of G columns from column col0 on.
constexpr int kMoWords = 36;  // 27 node ids, meta, 8 element ids
template <class T, int G>
__global__ void __launch_bounds__(128) mrhs_octet_pf_kernel(int64_t n, const uint32_t* __restrict__ ometa,
                                                            const uint32_t* __restrict__ oid,
                                                            const uint32_t* __restrict__ oelem,
                                                            const T* __restrict__ ca, const T* __restrict__ cb,
                                                            int R, int col0, int nb, const T* __restrict__ X,
                                                            T* __restrict__ Y) {
  constexpr int S = 32 / G;  // groups per warp
  __shared__ uint32_t slot[4 * S][2][kMoWords];
  const int gl = threadIdx.x % G, grp = threadIdx.x / G;
  const int64_t tasks = n * nb;
  const int64_t stride = (int64_t(gridDim.x) * blockDim.x) / G;
  auto fetch = [&](int64_t t, int sl) {
    if (t < tasks) {
      const int64_t o = t / nb;
      for (int k = gl; k < kMoWords; k += G) {
        const uint32_t* src = k < 27 ? oid + int64_t(k) * n + o : k == 27 ? ometa + o : oelem + int64_t(k - 28) * n + o;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&slot[grp][sl][k]))),
                     "l"(src)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // tw: the task of the warp's first group, the same for all its lanes
  int64_t t = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G, tw = t - grp % S;
  fetch(t, 0);
  for (int it = 0; tw < tasks; t += stride, tw += stride, ++it) {
    const int sl = it & 1;
    __syncwarp();  // every lane is done with the slot the next fetch overwrites
    fetch(t + stride, sl ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();  // the whole slot of this task has landed
    if (S > 1 && t >= tasks) continue;
    const uint32_t* W = slot[grp][sl];
    const int64_t o = t / nb;
    const int col = col0 + int(t - o * nb) * G + gl;
    const uint32_t m = W[27];
    uint32_t none = 0;
    T xv[27], yv[27];
#pragma unroll
    for (int p = 0; p < 27; ++p) {
      const uint32_t id = W[p];
      none |= id == kNoNode ? (1u << p) : 0u;
      xv[p] = id != kNoNode ? __ldg(X + int64_t(id) * R + col) : T(0);
    }
    octet_apply<T>(xv, yv, none, m, [&](int c, T& f1, T& f2) {
      if (ca) {
        const uint32_t e = W[28 + c];
        f1 *= __ldg(ca + e);
        f2 *= __ldg(cb + e);
      }
    });
    const uint32_t cm = ometa_cmask(m);
#pragma unroll
    for (int p = 0; p < 27; ++p) {
      const uint32_t id = W[p];
      if (id == kNoNode) continue;
      T* dst = Y + int64_t(id) * R + col;
      if (p == 13 && cm == 255u) *dst = yv[p];
      else if (yv[p] != T(0)) atomicAdd(dst, yv[p]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Two FP32 values in one 64-bit register, worked by the packed FP32
// instructions of sm_100 (add / sub / mul .f32x2): the octet arithmetic runs
// on two right-hand sides per instruction.
struct F2 {
  uint64_t v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ F2(double s) {
    const uint64_t u = __float_as_uint(float(s));
    v = (u << 32) | u;
  }
  __device__ __forceinline__ F2& operator+=(F2 b) {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(b.v));
    return *this;
  }
  __device__ __forceinline__ F2& operator*=(F2 b) {
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(b.v));
    return *this;
  }
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return a += b; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return a *= b; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ bool nonzero(F2 a) { return (a.v & 0x7fffffff7fffffffull) != 0ull; }

// The octet form with two right-hand sides per lane and G lanes per octet: X
// rows read as 8-byte pairs, Y rows added with 8-byte vector reductions, the
// element arithmetic on packed pairs.  Works nb blocks of 2 G columns from
// column col0 on (R and col0 even), G = 32, 16 or 8: with fewer lanes per octet
// a warp works 2 or 4 octets at once, whose missing children and hanging points
// differ, but at half the instructions per right-hand side.  64 columns are 711 M
// warp instructions, which fill 59 % of the issue slots (FMA pipe 46 %, L1 28 %,
// DRAM 21 %): dependent arithmetic with the 12 warps per SM that 168 registers
// leave.  On the 2.9M-element benchmark mesh, against one right-hand side per
// lane: 32 columns 634 and 817 us, 16 columns 330 and 444, 48 columns 989 and
// 1261; 64 columns 1140.
template <int G>
__global__ void __launch_bounds__(128) mrhs_octet_pair_kernel(int64_t n, const uint32_t* __restrict__ ometa,
                                                              const uint32_t* __restrict__ oid,
                                                              const uint32_t* __restrict__ oelem,
                                                              const float* __restrict__ ca,
                                                              const float* __restrict__ cb, int R, int col0, int nb,
                                                              const float* __restrict__ X, float* __restrict__ Y) {
  constexpr int S = 32 / G;  // groups per warp
  __shared__ uint32_t slot[4 * S][2][kMoWords];
  const int gl = threadIdx.x % G, grp = threadIdx.x / G;
  const int64_t tasks = n * nb;
  const int64_t stride = (int64_t(gridDim.x) * blockDim.x) / G;
  auto fetch = [&](int64_t t, int sl) {
    if (t < tasks) {
      const int64_t o = t / nb;
      for (int k = gl; k < kMoWords; k += G) {
        const uint32_t* src = k < 27 ? oid + int64_t(k) * n + o : k == 27 ? ometa + o : oelem + int64_t(k - 28) * n + o;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&slot[grp][sl][k]))),
                     "l"(src)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // tw: the task of the warp's first group, the same for all its lanes
  int64_t t = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G, tw = t - grp % S;
  fetch(t, 0);
  for (int it = 0; tw < tasks; t += stride, tw += stride, ++it) {
    const int sl = it & 1;
    __syncwarp();
    fetch(t + stride, sl ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    if (S > 1 && t >= tasks) continue;
    const uint32_t* W = slot[grp][sl];
    const int64_t o = t / nb;
    const int col = col0 + int(t - o * nb) * (2 * G) + 2 * gl;
    const uint32_t m = W[27];
    uint32_t none = 0;
    F2 xv[27], yv[27];
#pragma unroll
    for (int p = 0; p < 27; ++p) {
      const uint32_t id = W[p];
      none |= id == kNoNode ? (1u << p) : 0u;
      xv[p].v = id != kNoNode ? __ldg(reinterpret_cast<const unsigned long long*>(X + int64_t(id) * R + col))
                              : 0ull;
    }
    octet_apply<F2>(xv, yv, none, m, [&](int c, F2& f1, F2& f2) {
      if (ca) {
        const uint32_t e = W[28 + c];
        f1 *= F2(__ldg(ca + e));
        f2 *= F2(__ldg(cb + e));
      }
    });
    const uint32_t cm = ometa_cmask(m);
#pragma unroll
    for (int p = 0; p < 27; ++p) {
      const uint32_t id = W[p];
      if (id == kNoNode) continue;
      float* dst = Y + int64_t(id) * R + col;
      const float a = __uint_as_float(uint32_t(yv[p].v)), b = __uint_as_float(uint32_t(yv[p].v >> 32));
      if (p == 13 && cm == 255u)
        asm volatile("st.global.v2.f32 [%0], {%1, %2};" ::"l"(dst), "f"(a), "f"(b) : "memory");
      else if (nonzero(yv[p]))
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(dst), "f"(a), "f"(b) : "memory");
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <class T, int G>
void launch_octet(const dg_da* da, const T* ca, const T* cb, int R, int col0, int nb, const T* X, T* Y,
                  cudaStream_t s) {
  const OctetSet& O = da->octs;
  const int64_t warps = (O.n * nb + 32 / G - 1) / (32 / G);
  const unsigned grid = unsigned(std::min<int64_t>((warps + 3) / 4, int64_t(sm_count()) * 16));
  mrhs_octet_pf_kernel<T, G><<<grid, 128, 0, s>>>(O.n, O.meta.p, O.id.p, O.elem.p, ca, cb, R, col0, nb, X, Y);
}
template <int G>
void launch_pairs(const dg_da* da, const float* ca, const float* cb, int R, int col0, int nb, const float* X, float* Y,
                  cudaStream_t s) {
  const OctetSet& O = da->octs;
  const int64_t warps = (O.n * nb + 32 / G - 1) / (32 / G);
  const unsigned grid = unsigned(std::min<int64_t>((warps + 3) / 4, int64_t(sm_count()) * 16));
  mrhs_octet_pair_kernel<G><<<grid, 128, 0, s>>>(O.n, O.meta.p, O.id.p, O.elem.p, ca, cb, R, col0, nb, X, Y);
}

}  // namespace

// FP32: blocks of 64 columns by pairs, then 32, then 16 (2 and 4 octets per
// warp); FP64: 32 and 16.
template <class T>
dg_status mrhs_octet_apply(const dg_mat* A, const T* coef, const T* X, T* Y, int R, cudaStream_t s, bool zeroed) {
  const dg_da* da = A->da;
  const OctetSet& O = da->octs;
  DG_CHECK(A->kind == 0 && R % kRC == 0 && O.n > 0, DG_EINVAL, "multi-RHS octet operator: bad arguments");
  if (!zeroed) DG_CUDA(cudaMemsetAsync(Y, 0, sizeof(T) * size_t(da->N) * R, s));
  const T* ca = A->has_coef ? coef : nullptr;
  const T* cb = A->has_coef ? coef + da->E : nullptr;
  int col = 0;
  if constexpr (sizeof(T) == 4) {
    if (const int nb = R / 64) launch_pairs<32>(da, ca, cb, R, col, nb, X, Y, s);
    col = R & ~63;
    if ((R - col) & 32) launch_pairs<16>(da, ca, cb, R, col, 1, X, Y, s);
    col = R & ~31;
    if (R > col) launch_pairs<8>(da, ca, cb, R, col, 1, X, Y, s);
  } else {
    if (const int nb = R / 32) launch_octet<T, 32>(da, ca, cb, R, col, nb, X, Y, s);
    col = R & ~31;
    if (R > col) launch_octet<T, 16>(da, ca, cb, R, col, 1, X, Y, s);
  }
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
template dg_status mrhs_octet_apply<float>(const dg_mat*, const float*, const float*, float*, int, cudaStream_t,
                                           bool);
template dg_status mrhs_octet_apply<double>(const dg_mat*, const double*, const double*, double*, int, cudaStream_t,
                                            bool);

dg_status mrhs_apply(const dg_mat* A, const float* X, float* Y, int R, int split, cudaStream_t s) {
  dg_da* da = A->da;
  DG_CHECK(A->kind == 0, DG_EINVAL, "mat_mult_multi: scalar operator expected");
  DG_CHECK(R > 0 && R % kRC == 0, DG_EINVAL, "mat_mult_multi: nrhs must be a positive multiple of 16");
  DG_CHECK(split == 0 || split == 1 || split == 3 || split == 4 || split == 5, DG_EINVAL,
           "mat_mult_multi: split must be 0, 1, 3, 4 or 5");
  DG_CHECK((reinterpret_cast<uintptr_t>(X) & 15) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0, DG_EINVAL,
           "mat_mult_multi: X and Y must be 16-byte aligned");
  if (split >= 4) return mrhs_tc_apply(A, X, Y, R, split == 4 ? 1 : 3, s);
  // split 3 and 1 run the same kernels; split 0 keeps refusing what it refused
  // when they did not, so that a caller's error check still sees it
  if (split == 0)
    DG_CHECK(R % 32 == 0 && da->meshes == 1, DG_EINVAL,
             "mat_mult_multi: split 0 takes nrhs a multiple of 32 on one mesh");
  return mrhs_octet_apply<float>(A, A->has_coef ? A->coef32.p : nullptr, X, Y, R, s);
}

}  // namespace dg
