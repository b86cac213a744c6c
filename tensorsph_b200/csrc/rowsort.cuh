// Ascending sort of short uint32 rows in registers: W lanes share a row, each
// holding E entries; a warp takes 32 / W neighbouring rows at once.
//
// A bitonic network with the sorted position i = lane * E + register, so that
// exchanges at distances below E stay inside a lane (two min/max instructions)
// and only log2(W) (log2(W) + 1) / 2 of its steps are shuffles: three with the
// four lanes that rows of up to 64 entries get, six with eight lanes (up to
// 128), ten with 16.  Sixteen registers of entries are the most (with 32 the
// kernel takes 168 registers and loses more to idle warps than the shuffles
// cost).  Entries are loaded strided (any arrangement will do as input) and
// leave through shared memory, so that a row's stores are contiguous.
//
// What bounds it: instruction issue and, for pairs, the 16 bytes written per
// entry.  With a row per warp (entry = register * 32 + lane) the shuffles
// bound it, 40 for a 64-entry row against 6 here.  1.0 M rows of 38 entries,
// sorted and written out as pairs (0.77 GB moved), take 0.23 ms against 0.31,
// and 0.74 + 0.18 ms for a rank sort over shared memory and a pass that writes
// the pairs; 1.04 M 2-D rows of 10 entries in place 0.09 against 0.14 and 0.31.
#pragma once

#include "common.cuh"

namespace tsph {

constexpr int kGroupRow = 256;      // longest row rows_sort takes
constexpr int kMidRow = 1024;       // longest row a warp of rows_sort_rest takes
constexpr int kMediumRow = 8192;    // longest row a block sorts in shared memory
constexpr int kSortBlock = 128;
constexpr int kRestBlock = 512;

struct LongRows {
  int64_t* mid;      // rows of kGroupRow + 1 .. kMidRow entries
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

// A view of rows: where row r's entries are, the output position of its first
// one, how many there are.
struct CsrRows {
  uint32_t* vals;
  const int64_t* ptr;
  __device__ __forceinline__ uint32_t* src(int64_t r) const { return vals + ptr[r]; }
  __device__ __forceinline__ int64_t dst(int64_t r) const { return ptr[r]; }
  __device__ __forceinline__ int64_t len(int64_t r) const { return ptr[r + 1] - ptr[r]; }
};

// Outputs take (row, position, value).
struct AsEntries {
  uint32_t* vals;
  __device__ __forceinline__ void operator()(int64_t, int64_t pos, uint32_t v) const { vals[pos] = v; }
};

// (row, value) pairs; kWide: pairs is 16-byte aligned, one store each.
template <bool kWide>
struct AsPairs {
  int64_t* pairs;
  __device__ __forceinline__ void operator()(int64_t r, int64_t pos, uint32_t v) const {
    if (kWide) {
      *reinterpret_cast<longlong2*>(pairs + 2 * pos) = make_longlong2(r, static_cast<long long>(v));
    } else {
      pairs[2 * pos] = r;
      pairs[2 * pos + 1] = static_cast<int64_t>(v);
    }
  }
};

// Ascending over the W * E entries of a group of W lanes, at i = gl * E + r.
template <int E, int W>
__device__ __forceinline__ void bitonic_regs(uint32_t (&v)[E], int gl) {
#pragma unroll
  for (int k = 2; k <= W * E; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j < E) {
#pragma unroll
        for (int r = 0; r < E; ++r) {
          if (r & j) continue;
          const bool asc = ((gl * E + r) & k) == 0;  // known at compile time for k < E
          const uint32_t a = v[r], b = v[r | j];
          v[r] = asc ? min(a, b) : max(a, b);
          v[r | j] = asc ? max(a, b) : min(a, b);
        }
      } else {
        const bool keep_low = ((gl & (j / E)) == 0) == (((gl * E) & k) == 0);
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j / E);
          v[r] = keep_low ? min(v[r], o) : max(v[r], o);
        }
      }
    }
  }
}

// 32 / W rows from r0 on, every one of at most W * E entries; all lanes of the
// warp take part.  buf: 32 * (E + 1) words of the warp's own.
template <int E, int W, class Rows, class Out>
__device__ __forceinline__ void sort_group(const Rows& rows, int64_t r0, int64_t n, const Out& out,
                                           uint32_t* buf) {
  const int lane = threadIdx.x & 31, gl = lane & (W - 1), g = lane / W;
  const int64_t r = r0 + g;
  const int len = r < n ? static_cast<int>(rows.len(r)) : 0;
  const uint32_t* src = r < n ? rows.src(r) : nullptr;
  const int64_t dst = r < n ? rows.dst(r) : 0;
  uint32_t v[E];
#pragma unroll
  for (int i = 0; i < E; ++i) v[i] = i * W + gl < len ? src[i * W + gl] : 0xffffffffu;
  bitonic_regs<E, W>(v, gl);
  // sorted position p of group g at ((g * W + p / E) * (E + 1) + p % E): one
  // spare word per lane keeps the stores off each other's banks
  __syncwarp();
#pragma unroll
  for (int i = 0; i < E; ++i) buf[lane * (E + 1) + i] = v[i];
  __syncwarp();
#pragma unroll 1
  for (int q = 0; q < 32 / W; ++q) {
    const int lq = __shfl_sync(0xffffffffu, len, q * W);
    const int64_t dq = __shfl_sync(0xffffffffu, dst, q * W);
    for (int p = lane; p < lq; p += 32) out(r0 + q, dq + p, buf[(q * W + p / E) * (E + 1) + p % E]);
  }
}

// Rows with those beyond kGroupRow left out.
template <class Rows>
struct Bounded {
  const Rows& rows;
  __device__ __forceinline__ uint32_t* src(int64_t r) const { return rows.src(r); }
  __device__ __forceinline__ int64_t dst(int64_t r) const { return rows.dst(r); }
  __device__ __forceinline__ int64_t len(int64_t r) const {
    const int64_t l = rows.len(r);
    return l <= kGroupRow ? l : 0;
  }
};

// What a warp does besides for its rows r0 .. r0 + 7 (below n); all lanes call it.
template <class Rows>
__device__ __forceinline__ void beside_rows(const Rows&, int64_t, int64_t) {}

// The rows may lie where the output goes: a row is read whole before any of it
// is written, and rows do not overlap.
template <class Rows, class Out>
__global__ void __launch_bounds__(kSortBlock, 8) rows_sort(Rows rows, int64_t n, Out out, LongRows lists) {
  __shared__ uint32_t buf[kSortBlock / 32][32 * 17];
  const int lane = threadIdx.x & 31;
  uint32_t* mine = buf[threadIdx.x >> 5];
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * kSortBlock) >> 5;
  for (int64_t w = (static_cast<int64_t>(blockIdx.x) * kSortBlock + threadIdx.x) >> 5; 8 * w < n; w += warps) {
    const int64_t r0 = 8 * w, r = r0 + (lane & 7);
    const int64_t len = r < n ? rows.len(r) : 0;
    beside_rows(rows, r0, n);
    int64_t longest = len;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
    if (longest == 0) continue;
    if (longest <= 8)
      sort_group<2, 4>(rows, r0, n, out, mine);
    else if (longest <= 16)
      sort_group<4, 4>(rows, r0, n, out, mine);
    else if (longest <= 32)
      sort_group<8, 4>(rows, r0, n, out, mine);
    else if (longest <= 64)
      sort_group<16, 4>(rows, r0, n, out, mine);
    else {
      // a row beyond kGroupRow is listed and left empty here
      if (lane < 8 && len > kGroupRow) {
        if (len <= kMidRow)
          lists.mid[atomicAdd(&lists.counts[0], 1ull)] = r;
        else
          lists.big[atomicAdd(&lists.counts[1], 1ull)] = r;
      }
      const Bounded<Rows> bounded{rows};
      if (longest <= 128) {
#pragma unroll 1
        for (int h = 0; h < 8; h += 4) sort_group<16, 8>(bounded, r0 + h, n, out, mine);
      } else {
#pragma unroll 1
        for (int h = 0; h < 8; h += 2) sort_group<16, 16>(bounded, r0 + h, n, out, mine);
      }
    }
  }
}

// The rows beyond kGroupRow: mid rows by one warp each (entry = register * 32 +
// lane of the sorted order, as above with 32 lanes), longer ones by one block
// each, in shared memory up to kMediumRow and beyond it where they lie: stretches
// of kMediumRow in shared memory, and directly only the steps between stretches
// (21 of the 190 steps of 300 k entries, which bound such a row: 32.4 ms with all of
// them in global memory).  The network is the all-ascending form (the first step of
// each merge pairs t with t ^ (k - 1)), so the minimum always lands on the lower
// index and the virtual +inf padding beyond `len` never moves.
template <class Rows, class Out>
__global__ void __launch_bounds__(kRestBlock, 1) rows_sort_rest(Rows rows, Out out, LongRows lists) {
  __shared__ uint32_t buf[kMediumRow];
  const int64_t mids = static_cast<int64_t>(lists.counts[0]), bigs = static_cast<int64_t>(lists.counts[1]);
  const int lane = threadIdx.x & 31;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * kRestBlock) >> 5;
  for (int64_t q = (static_cast<int64_t>(blockIdx.x) * kRestBlock + threadIdx.x) >> 5; q < mids; q += warps) {
    const int64_t r = lists.mid[q], dst = rows.dst(r);
    const uint32_t* src = rows.src(r);
    const int len = static_cast<int>(rows.len(r));
    uint32_t v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = i * 32 + lane < len ? src[i * 32 + lane] : 0xffffffffu;
    bitonic_regs<32, 32>(v, lane);
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (lane * 32 + i < len) out(r, dst + lane * 32 + i, v[i]);
  }
  // the steps of merge k at distances j, j / 2, .., 1 over buf[0, p2)
  auto merge = [&](int k, int j, int p2) {
    for (; j > 0; j >>= 1) {
      const int mask = 2 * j == k ? k - 1 : j;
      for (int t = threadIdx.x; t < p2; t += blockDim.x) {
        const int u = t ^ mask;
        if (u > t) {
          const uint32_t x = buf[t], y = buf[u];
          if (x > y) { buf[t] = y; buf[u] = x; }
        }
      }
      __syncthreads();
    }
  };
  auto load = [&](const uint32_t* a, int64_t len, int p2) {
    for (int t = threadIdx.x; t < p2; t += blockDim.x) buf[t] = t < len ? a[t] : 0xffffffffu;
    __syncthreads();
  };
  for (int64_t q = blockIdx.x; q < bigs; q += gridDim.x) {
    const int64_t r = lists.big[q], dst = rows.dst(r), len = rows.len(r);
    uint32_t* a = rows.src(r);
    int64_t p2 = 1;
    while (p2 < len) p2 <<= 1;
    if (len <= kMediumRow) {
      load(a, len, static_cast<int>(p2));
      for (int k = 2; k <= p2; k <<= 1) merge(k, k >> 1, static_cast<int>(p2));
      for (int t = threadIdx.x; t < len; t += blockDim.x) out(r, dst + t, buf[t]);
    } else {
      auto stretches = [&](auto&& steps) {
        for (int64_t b = 0; b < len; b += kMediumRow) {
          load(a + b, len - b, kMediumRow);
          steps();
          for (int t = threadIdx.x; t < kMediumRow && t < len - b; t += blockDim.x) a[b + t] = buf[t];
          __syncthreads();
        }
      };
      stretches([&] {
        for (int k = 2; k <= kMediumRow; k <<= 1) merge(k, k >> 1, kMediumRow);
      });
      for (int64_t k = 2 * kMediumRow; k <= p2; k <<= 1) {
        for (int64_t j = k >> 1; j >= kMediumRow; j >>= 1) {
          const int64_t mask = (j == (k >> 1)) ? (k - 1) : j;
          for (int64_t t = threadIdx.x; t < p2; t += blockDim.x) {
            const int64_t u = t ^ mask;
            if (u > t && t < len && u < len) {
              const uint32_t x = a[t], y = a[u];
              if (x > y) { a[t] = y; a[u] = x; }
            }
          }
          __syncthreads();
        }
        stretches([&] { merge(0, kMediumRow >> 1, kMediumRow); });
      }
      for (int64_t t = threadIdx.x; t < len; t += blockDim.x) out(r, dst + t, a[t]);
    }
    __syncthreads();
  }
}

// Sort the n rows of `rows` and hand them to out.  `longest` bounds
// the length of a row (or the entries of all rows together): up to kGroupRow the
// second kernel is not launched.  Scratch: segsort_scratch_bytes(n).
template <class Rows, class Out>
int sort_rows(Rows rows, int64_t n, int64_t longest, Out out, void* scratch, cudaStream_t s) {
  if (n <= 0) return TSPH_OK;
  const LongRows lists = long_rows(scratch, n);
  const bool rest = longest > kGroupRow;
  if (rest) TSPH_CUDA_CHECK(cudaMemsetAsync(lists.counts, 0, 2 * sizeof(unsigned long long), s));
  rows_sort<Rows, Out><<<grid_for((n + 7) / 8, kSortBlock / 32, 148 * 64), kSortBlock, 0, s>>>(rows, n, out, lists);
  TSPH_LAUNCH_CHECK();
  if (rest) {
    rows_sort_rest<Rows, Out><<<148, kRestBlock, 0, s>>>(rows, out, lists);
    TSPH_LAUNCH_CHECK();
  }
  return TSPH_OK;
}

}  // namespace tsph
