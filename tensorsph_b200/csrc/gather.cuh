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

// Calls f(lanes per row) for rows of a D-dimensional cloud.  Device time of the
// three passes of an rhs (density, diffusion, force; FP32, then FP64; us):
//   2-D, ~20 entries    L = 1        2        4
//       5 k rows        30  35   21  24   16  18
//      24 k             33  38   23  26   18  21
//      36 k             34  40   25  28   21  28
//      49 k             35  41   26  31   27  36
//     250 k             79  98   73  98   92 124
//     400 k            108 150  108 148
//     550 k            140 200  144 204
//     1.0 M            243 344  252 359
//   3-D, ~80 entries    L = 2        4        8
//       4 k rows        65  73   37  42   24  26
//      23 k             67  79   42  50   37  54
//      33 k             69  82   49  70   50  66
//      48 k             77  90   68  95   63  90
//      81 k             96 150   94 135   95 140
//     161 k            177 250  168 255
//     201 k            216 318  210 323
//     420 k            424 642  441 680
// (threed's passes alike, FP64: 24 k rows 101 / 102 with four / eight lanes, 36 k
// 160 / 135, 64 k 210 / 209.)  One line serves both dtypes and every pass: four lanes
// in 2-D pay up to 36 k rows in FP64 and 45 k in FP32, and cost at most 5 us of a
// ~110 us call between there and the line; eight in 3-D are the fastest or within
// 4 us up to theirs.
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
