// Several lanes per gather row.
//
// The row kernels of the drop-in passes sum over a particle's neighbours.  L
// neighbouring lanes share a row: lane l takes entries l, l + L, ..., and the
// lanes' sums are combined in a fixed order, so a result depends on the row and
// on L only, not on the launch.  That shortens the chains of dependent loads
// and of FP64 additions by L and lets a few thousand rows fill the chip; it
// costs the combination (with_lanes: where the lines lie).  Reading a row's
// entries 16 bytes at a time with masked ends was slower at every L (1.0 M 2-D
// FP32 rows: 415 us against 330 for the three passes): the rows stay in the L1,
// and instruction issue bounds the passes.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace tsph {

constexpr uint32_t kIndexMask = 0x7fffffffu;
constexpr int kGatherBlock = 128;

template <class T>
struct alignas(4 * sizeof(T)) Q4 {
  T x, y, z, w;
};

template <class T>
struct alignas(2 * sizeof(T)) Q2 {
  T x, y;
};

// This thread's row, lane and the lanes of its row in the warp.
template <int L>
struct RowLanes {
  int64_t row;
  int lane;
  unsigned group;
  __device__ __forceinline__ RowLanes()
      : row((blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / L),
        lane(threadIdx.x & (L - 1)),
        group((L == 32 ? 0xffffffffu : (1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1))) {}
  // The sum over the row's lanes, in every lane; total() with its compensation.
  template <class T>
  __device__ __forceinline__ CSum<T> total(CSum<T> s) const;
  template <class T>
  __device__ __forceinline__ T sum(CSum<T> s) const {
    return total(s).value();
  }
  // Calls use(entry) for this lane's part of the row's entries [beg, end).
  template <class Use>
  __device__ __forceinline__ void walk(const uint32_t* __restrict__ ent, int64_t beg, int64_t end, Use&& use) const {
    const uint32_t* __restrict__ row_ent = ent + beg;
    const int len = static_cast<int>(end - beg);
#pragma unroll 2
    for (int k = lane; k < len; k += L) use(row_ent[k]);
  }
  // The same with the next two entries on their way while two are used, for the
  // passes that wait on their gathers: a term's chain is one load instead of two
  // (FP64, 3-D, us a launch: 480 k rows, colour 219 -> 188, gradient 231 -> 194,
  // kappa 241 -> 219; 262 k rows, density 102 -> 83, moments 143 -> 117, diffusion
  // 179 -> 156; FP32 densities 54 -> 50 and 56 -> 51).  The passes bound by issue or
  // by registers lose by it (FP64 3-D force 193 -> 210, FP32 diffusion 79 -> 85).
  // Loading the records as well a step ahead was no faster (202, 195, 210).
  template <class Use>
  __device__ __forceinline__ void walk_ahead(const uint32_t* __restrict__ ent, int64_t beg, int64_t end,
                                             Use&& use) const {
    const uint32_t* __restrict__ row_ent = ent + beg;
    const int len = static_cast<int>(end - beg);
    int k = lane;
    if (k >= len) return;
    uint32_t e0 = row_ent[k], e1 = row_ent[min(k + L, len - 1)];
    for (; k + L < len; k += 2 * L) {
      const uint32_t n0 = row_ent[min(k + 2 * L, len - 1)], n1 = row_ent[min(k + 3 * L, len - 1)];
      use(e0);
      use(e1);
      e0 = n0;
      e1 = n1;
    }
    if (k < len) use(e0);
  }
};

template <class T>
__device__ __forceinline__ void join(CSum<T>& s, unsigned group, int o) {
  s.s += __shfl_xor_sync(group, s.s, o);
}
template <>
__device__ __forceinline__ void join<float>(CSum<float>& s, unsigned group, int o) {
  const float os = __shfl_xor_sync(group, s.s, o), oc = __shfl_xor_sync(group, s.c, o);
  s.add(os);
  s.c = __fadd_rn(s.c, oc);
}

template <int L>
template <class T>
__device__ __forceinline__ CSum<T> RowLanes<L>::total(CSum<T> s) const {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) join(s, group, o);
  return s;
}

// Blocks for n rows of L lanes.
inline unsigned row_grid(int64_t n, int lanes, int block = kGatherBlock) {
  const int64_t g = (n * lanes + block - 1) / block;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

// Calls f(lanes per row) for rows of a D-dimensional cloud.  The lines lie where
// whole rhs passes (density, diffusion, force; FP32, then FP64; us) cross:
//   2-D, ~20 entries    L = 1        2        4
//       5 k rows       51  59    44  44    37  41
//      60 k            58  66    49  54    57  64
//     250 k            99 124    91 119   130 160
//     1.0 M           275 409   297 414   447 613
//   3-D, ~80 entries    L = 2        4        8
//       5 k rows      110 122    74  81    58  62
//      24 k           114 129    78  89    76  96
//      82 k           140 201   132 178   153 203
//     241 k           313 486   324 491   408 604
// (L = 4 in 2-D and 8 in 3-D measured with divisions in the terms.)
template <int D, class F>
int with_lanes(int64_t rows, F&& f) {
  if (D == 3) {
    if (rows <= 49152) return f(std::integral_constant<int, 8>{});
    if (rows <= 196608) return f(std::integral_constant<int, 4>{});
    return f(std::integral_constant<int, 2>{});
  }
  if (rows <= 49152) return f(std::integral_constant<int, 4>{});
  if (rows <= 524288) return f(std::integral_constant<int, 2>{});
  return f(std::integral_constant<int, 1>{});
}

}  // namespace tsph
