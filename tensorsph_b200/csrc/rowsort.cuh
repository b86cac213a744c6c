// Ascending sort of short uint32 rows, one row per warp (or two rows of up to
// 16 entries per warp), held in registers as a bitonic network: entry i of a
// row sits in register i / W of lane i % W of its W-lane group, so exchanges
// at distances below W are shuffles and the others stay inside a lane.
//
// What bounds it: instruction issue and the latency of the row bounds, not
// bytes.  A row of 39 entries (the one-sided 3-D list at 2.6 dx) takes a
// 64-entry network, 21 exchanges of two registers, against 39 x 2 compare
// steps per lane of a rank sort over shared memory: 480 k rows of 39 entries
// sort in 0.15 ms against 0.32.
//
// Rows is a view: beg(r) and len(r).  Out takes (r, position, value).  Rows
// longer than kWarpRow are appended to `lists` for rows_sort_rest.
#pragma once

#include "common.cuh"

namespace tsph {

constexpr int kWarpRow = 256;       // longest row a warp sorts in eight registers a lane
constexpr int kMidRow = 1024;       // longest row a warp sorts in 32
constexpr int kMediumRow = 8192;    // longest row a block sorts in shared memory
constexpr int kSortBlock = 256;
constexpr int kRestBlock = 512;

struct LongRows {
  int64_t* mid;      // rows of kWarpRow + 1 .. kMidRow entries
  int64_t* big;      // longer ones
  unsigned long long* counts;  // [0] mid, [1] big
};

inline LongRows long_rows(void* scratch, int64_t rows) {
  char* sc = static_cast<char*>(scratch);
  LongRows l;
  l.counts = reinterpret_cast<unsigned long long*>(sc);
  l.mid = reinterpret_cast<int64_t*>(sc + 256);
  l.big = reinterpret_cast<int64_t*>(sc + 256 + align_up((rows + 1) * sizeof(int64_t)));
  return l;
}

// Rows of a CSR table.
struct CsrRows {
  const int64_t* ptr;
  __device__ __forceinline__ int64_t beg(int64_t r) const { return ptr[r]; }
  __device__ __forceinline__ int64_t len(int64_t r) const { return ptr[r + 1] - ptr[r]; }
};

// Back into the array the rows came from.
struct InPlace {
  uint32_t* vals;
  static constexpr bool kAll = false;  // rows of one entry are already in place
  __device__ __forceinline__ void operator()(int64_t, int64_t pos, uint32_t v) const { vals[pos] = v; }
};

// E registers x W lanes, ascending over each group of W lanes.
template <int E, int W>
__device__ __forceinline__ void bitonic_regs(uint32_t (&v)[E], int gl) {
#pragma unroll
  for (int k = 2; k <= W * E; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j < W) {
        const bool lower = (gl & j) == 0;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const bool asc = ((r * W + gl) & k) == 0;
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j);
          v[r] = (lower == asc) ? min(v[r], o) : max(v[r], o);
        }
      } else {
        const int jr = j / W;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          if (r & jr) continue;
          const bool asc = ((r * W + gl) & k) == 0;
          const uint32_t a = v[r], b = v[r | jr];
          v[r] = asc ? min(a, b) : max(a, b);
          v[r | jr] = asc ? max(a, b) : min(a, b);
        }
      }
    }
  }
}

template <int E, int W, class Out>
__device__ __forceinline__ void sort_row(const uint32_t* __restrict__ vals, int64_t r, int64_t beg, int len,
                                         int gl, const Out& out) {
  uint32_t v[E];
#pragma unroll
  for (int i = 0; i < E; ++i) v[i] = i * W + gl < len ? vals[beg + i * W + gl] : 0xffffffffu;
  bitonic_regs<E, W>(v, gl);
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (i * W + gl < len) out(r, beg + i * W + gl, v[i]);
}

// `vals` is not __restrict__: with InPlace it is also the output, and every
// row is read into registers before any of it is written.
template <class Rows, class Out>
__global__ void __launch_bounds__(kSortBlock) rows_sort(const uint32_t* vals, Rows rows, int64_t n, Out out,
                                                        LongRows lists) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * kSortBlock) >> 5;
  for (int64_t w = (static_cast<int64_t>(blockIdx.x) * kSortBlock + threadIdx.x) >> 5; 2 * w < n; w += warps) {
    const int64_t r0 = 2 * w;
    const bool two = r0 + 1 < n;
    // half a warp per row of the pair: lengths of both rows in every lane
    const int64_t b0 = rows.beg(r0), l0 = rows.len(r0);
    const int64_t b1 = two ? rows.beg(r0 + 1) : 0, l1 = two ? rows.len(r0 + 1) : 0;
    if (l0 <= 16 && l1 <= 16) {
      const bool second = lane >= 16;
      const int len = static_cast<int>(second ? l1 : l0);
      if ((l0 > l1 ? l0 : l1) > (Out::kAll ? 0 : 1))
        sort_row<1, 16>(vals, second ? r0 + 1 : r0, second ? b1 : b0, len, lane & 15, out);
      continue;
    }
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      const int64_t r = r0 + k, beg = k ? b1 : b0, len = k ? l1 : l0;
      const int n32 = static_cast<int>(len);
      if (len <= (Out::kAll ? 0 : 1)) continue;
      if (len <= 32)
        sort_row<1, 32>(vals, r, beg, n32, lane, out);
      else if (len <= 64)
        sort_row<2, 32>(vals, r, beg, n32, lane, out);
      else if (len <= 128)
        sort_row<4, 32>(vals, r, beg, n32, lane, out);
      else if (len <= kWarpRow)
        sort_row<8, 32>(vals, r, beg, n32, lane, out);
      else if (lane == 0) {
        if (len <= kMidRow)
          lists.mid[atomicAdd(&lists.counts[0], 1ull)] = r;
        else
          lists.big[atomicAdd(&lists.counts[1], 1ull)] = r;
      }
    }
  }
}

// The rows beyond kWarpRow: mid rows by one warp each, longer ones by one
// block each, in shared memory up to kMediumRow and beyond it directly in
// global memory.  The global network is the all-ascending form (the first
// step of each merge pairs t with t ^ (k - 1)), so the minimum always lands
// on the lower index and the virtual +inf padding beyond `len` never moves.
template <class Rows, class Out>
__global__ void __launch_bounds__(kRestBlock) rows_sort_rest(uint32_t* vals, Rows rows, Out out, LongRows lists) {
  __shared__ uint32_t buf[kMediumRow];
  const int lane = threadIdx.x & 31;
  const int64_t mids = static_cast<int64_t>(lists.counts[0]), bigs = static_cast<int64_t>(lists.counts[1]);
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * kRestBlock) >> 5;
  for (int64_t q = (static_cast<int64_t>(blockIdx.x) * kRestBlock + threadIdx.x) >> 5; q < mids; q += warps) {
    const int64_t r = lists.mid[q], beg = rows.beg(r);
    const int len = static_cast<int>(rows.len(r));
    if (len <= 512)
      sort_row<16, 32>(vals, r, beg, len, lane, out);
    else
      sort_row<32, 32>(vals, r, beg, len, lane, out);
  }
  for (int64_t q = blockIdx.x; q < bigs; q += gridDim.x) {
    const int64_t r = lists.big[q], beg = rows.beg(r), len = rows.len(r);
    int64_t p2 = 1;
    while (p2 < len) p2 <<= 1;
    if (len <= kMediumRow) {
      for (int t = threadIdx.x; t < p2; t += blockDim.x) buf[t] = t < len ? vals[beg + t] : 0xffffffffu;
      __syncthreads();
      for (int k = 2; k <= p2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
          for (int t = threadIdx.x; t < p2; t += blockDim.x) {
            const int ixj = t ^ j;
            if (ixj > t) {
              const bool up = (t & k) == 0;
              const uint32_t x = buf[t], y = buf[ixj];
              if ((x > y) == up) { buf[t] = y; buf[ixj] = x; }
            }
          }
          __syncthreads();
        }
      }
      for (int t = threadIdx.x; t < len; t += blockDim.x) out(r, beg + t, buf[t]);
    } else {
      uint32_t* a = vals + beg;
      for (int64_t k = 2; k <= p2; k <<= 1) {
        for (int64_t j = k >> 1; j > 0; j >>= 1) {
          const int64_t mask = (j == (k >> 1)) ? (k - 1) : j;
          for (int64_t t = threadIdx.x; t < p2; t += blockDim.x) {
            const int64_t ixj = t ^ mask;
            if (ixj > t && t < len && ixj < len) {
              const uint32_t x = a[t], y = a[ixj];
              if (x > y) { a[t] = y; a[ixj] = x; }
            }
          }
          __syncthreads();
        }
      }
      if (Out::kAll)
        for (int64_t t = threadIdx.x; t < len; t += blockDim.x) out(r, beg + t, a[t]);
    }
    __syncthreads();
  }
}

// Sort the n rows of `rows` in vals and hand them to out.  `entries` bounds
// the entries of all rows together: below kWarpRow + 1 no row can be long, and
// the second kernel is not launched.  Scratch: segsort_scratch_bytes(n).
template <class Rows, class Out>
int sort_rows(uint32_t* vals, Rows rows, int64_t n, int64_t entries, Out out, void* scratch, cudaStream_t s) {
  if (n <= 0) return TSPH_OK;
  const LongRows lists = long_rows(scratch, n);
  const bool rest = entries > kWarpRow;
  if (rest) TSPH_CUDA_CHECK(cudaMemsetAsync(lists.counts, 0, 2 * sizeof(unsigned long long), s));
  rows_sort<Rows, Out><<<grid_for((n + 1) / 2, kSortBlock / 32, 148 * 16), kSortBlock, 0, s>>>(vals, rows, n, out,
                                                                                              lists);
  TSPH_LAUNCH_CHECK();
  if (rest) {
    rows_sort_rest<Rows, Out><<<148 * 2, kRestBlock, 0, s>>>(vals, rows, out, lists);
    TSPH_LAUNCH_CHECK();
  }
  return TSPH_OK;
}

}  // namespace tsph
