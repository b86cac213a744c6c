// Pair list -> symmetric, row-sorted gather list.
//
// The reference scatters every pair twice with index_add (once into i, once
// into j).  The B200 path turns the same list into per-particle rows so that
// each particle gathers its own sums in registers: no atomics in any
// floating-point accumulation, a fixed summation order, and coalesced
// per-particle writes.  Entry = neighbour index | (1u << 31) when the row is
// the pair's second element (the threed viscous operator weights a pair by
// the mass of its second element, operators3.py:137-160).
//
// A row is its first-element entries ascending, then its second-element ones.
// Two routes build it:
//
//   sorted list (what the searches of this library return, and the
//   reference's): the pairs of row i are one run of the list, already in
//   order, so only the second halves need counting, collecting and sorting:
//     A  list_place  run boundaries; one atomic per pair counts row j's second
//                    halves and hands out a place among the row's slots, where
//                    i goes at once
//     scan of the degrees
//     B  rows_sort   the second halves from the slots to their place, sorted;
//                    the same warp copies the rows' runs (coalesced)
//     A row with more second halves than slots is filled by another pass over
//     the list (list_rest) and sorted where it lies.
//   any other list: two atomics per pair to count, two to fill, rows sorted whole.
//
// What bounds the first route: the L2 atomics of A (one per pair) with the
// scattered 4-byte stores behind them, instruction issue and the copies' loads
// in B.  18.6 M pairs of a periodic column (480 k rows): A 0.17, scan 0.01,
// B 0.14 ms; counting first (0.13), filling by another pass over the list (0.15)
// and sorting (0.11) took 0.41, the second route with a rank sort of whole rows
// 1.2 ms.  13.1 M pairs of a block in mixed order 0.31 against 0.45, 10.6 M of a
// 2-D column (1.04 M rows) 0.23 against 0.26.  The copies in a launch of their own
// (0.09) or 32 pairs at a time (0.07 more than 128) lose to B's.
#include <algorithm>

#include "common.cuh"
#include "rowsort.cuh"

namespace tsph {
namespace {

constexpr uint32_t kSecond = 0x80000000u;
constexpr int kBlock = 256;
// The loads of a warp are one contiguous 512-byte run.  A thread of list_place takes
// two pairs, so that two atomics are on their way (18.6 M pairs 178 -> 166 us, 10.6 M
// 2-D ones 97 -> 85, the same in mixed order; four: 170, 94 and 6 % slower there).
constexpr int kPairs = 2;

enum { kBad = 1, kUnsorted = 2, kOver = 4 };  // kOver: a row has more second halves than slots

// kWide: the list starts on a 16-byte boundary (one load per pair).
template <bool kWide>
__device__ __forceinline__ longlong2 ld_pair(const int64_t* __restrict__ pairs, int64_t p) {
  if (kWide) return *reinterpret_cast<const longlong2*>(pairs + 2 * p);
  return make_longlong2(pairs[2 * p], pairs[2 * p + 1]);
}

// Lists of up to this many pairs also count the rows' degrees in A, so that an
// unsorted one needs no second count (whole calls: 500 pairs 92 -> 70 us, 100 k 102 ->
// 82; sorted ones the same within 1 us up to here).  A longer unsorted one pays A for
// finding out: 1.0 M pairs 145 us, 140 by the general route alone.
constexpr int64_t kSmallList = 131072;

// A: with the list found unsorted by an earlier block the rest of the grid only
// looks at the indices' range (an unsorted list is seen within its first pairs), so
// that the host waits once for either route.  The read of `found` goes through the
// L1, so a block may still miss the flag; it is no more than a short cut, and the
// host reads the flags after the kernel.
template <bool kWide, bool kDegrees>
__global__ void __launch_bounds__(kBlock) list_place(const int64_t* __restrict__ pairs, int64_t npairs,
                                                     int64_t nrows, int2* __restrict__ run,
                                                     int32_t* __restrict__ deg, unsigned int* __restrict__ second,
                                                     uint32_t* __restrict__ slots, unsigned int per_row,
                                                     unsigned int* found) {
  const bool range_only = !kDegrees && (*found & kUnsorted);
  const int64_t p0 = static_cast<int64_t>(blockIdx.x) * (kPairs * kBlock) + threadIdx.x;
  longlong2 me[kPairs], prev[kPairs];
#pragma unroll
  for (int u = 0; u < kPairs; ++u) {
    const int64_t p = p0 + u * kBlock;
    me[u] = p < npairs ? ld_pair<kWide>(pairs, p) : make_longlong2(-1, -1);
    prev[u] = !range_only && p > 0 && p < npairs ? ld_pair<kWide>(pairs, p - 1) : make_longlong2(-1, -1);
  }
  unsigned int s[kPairs];
#pragma unroll
  for (int u = 0; u < kPairs; ++u) {
    const int64_t p = p0 + u * kBlock;
    s[u] = 0xffffffffu;
    if (p >= npairs) continue;
    const int64_t i = me[u].x, j = me[u].y;
    if (i < 0 || j < 0 || i >= nrows || j >= nrows) {
      atomicOr(found, kBad);
      continue;
    }
    if (range_only) continue;
    if (kDegrees) {
      atomicAdd(&deg[i], 1);
      atomicAdd(&deg[j], 1);
    }
    if (prev[u].x > i || (prev[u].x == i && prev[u].y > j)) {
      atomicOr(found, kUnsorted);
      continue;
    }
    s[u] = atomicAdd(&second[j], 1u);
    if (prev[u].x != i) {
      run[i].x = static_cast<int>(p);
      if (prev[u].x >= 0 && prev[u].x < nrows) run[prev[u].x].y = static_cast<int>(p);
    }
    if (p == npairs - 1) run[i].y = static_cast<int>(npairs);
  }
#pragma unroll
  for (int u = 0; u < kPairs; ++u) {
    if (s[u] == 0xffffffffu) continue;
    if (s[u] < per_row)
      slots[me[u].y * per_row + s[u]] = static_cast<uint32_t>(me[u].x) | kSecond;
    else if (s[u] == per_row)
      atomicOr(found, kOver);
  }
}

__global__ void list_rows(const int2* __restrict__ run, const unsigned int* __restrict__ second, int64_t nrows,
                          int32_t* __restrict__ deg) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r < nrows) deg[r] = run[r].y - run[r].x + static_cast<int32_t>(second[r]);
}

// The second halves of the rows without enough slots, in any order to where they belong.
template <bool kWide>
__global__ void __launch_bounds__(kBlock) list_rest(const int64_t* __restrict__ pairs, int64_t npairs,
                                                    const int2* __restrict__ run, const int64_t* __restrict__ rowptr,
                                                    const unsigned int* __restrict__ second, unsigned int per_row,
                                                    unsigned int* __restrict__ placed,
                                                    uint32_t* __restrict__ entries) {
  const int64_t p = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (p >= npairs) return;
  const longlong2 me = ld_pair<kWide>(pairs, p);
  if (second[me.y] <= per_row) return;
  const int2 rj = run[me.y];
  entries[rowptr[me.y] + (rj.y - rj.x) + atomicAdd(&placed[me.y], 1u)] = static_cast<uint32_t>(me.x) | kSecond;
}

// The second-element halves of the rows.
template <bool kWide>
struct SecondHalves {
  uint32_t* entries;
  const int64_t* rowptr;
  const int2* run;
  const unsigned int* second;
  uint32_t* slots;
  unsigned int per_row;
  const int64_t* pairs;
  __device__ __forceinline__ int64_t dst(int64_t r) const { return rowptr[r] + (run[r].y - run[r].x); }
  __device__ __forceinline__ uint32_t* src(int64_t r) const {
    return second[r] <= per_row ? slots + r * per_row : entries + dst(r);
  }
  __device__ __forceinline__ int64_t len(int64_t r) const { return second[r]; }
};

// The first halves: the runs of rows r0 .. r0 + 7 are one stretch of the list.
template <bool kWide>
__device__ __forceinline__ void beside_rows(const SecondHalves<kWide>& rows, int64_t r0, int64_t n) {
  const int lane = threadIdx.x & 31;
  const int64_t r = r0 + (lane & 7);
  const int2 q = r < n ? rows.run[r] : make_int2(0, 0);
  const long long shift = r < n ? rows.rowptr[r] - q.x : 0;
  int first = q.y > q.x ? q.x : 0x7fffffff, last = q.y > q.x ? q.y : 0;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
    last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
  }
  // (eight rows without a run: first lies beyond last)
  for (int64_t base = first; base < last; base += 128) {
    const int64_t p0 = base + lane;
    longlong2 me[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) me[u] = ld_pair<kWide>(rows.pairs, min(p0 + 32 * u, static_cast<int64_t>(last - 1)));
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long to = __shfl_sync(0xffffffffu, shift, static_cast<int>(me[u].x - r0));
      if (p0 + 32 * u < last) rows.entries[to + p0 + 32 * u] = static_cast<uint32_t>(me[u].y);
    }
  }
}

__global__ void csr_degree(const int64_t* __restrict__ pairs, int64_t npairs, int64_t nrows,
                           int32_t* __restrict__ deg, unsigned int* __restrict__ found) {
  for (int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; p < npairs;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t i = pairs[2 * p], j = pairs[2 * p + 1];
    if (i < 0 || j < 0 || i >= nrows || j >= nrows) {
      atomicOr(found, kBad);
      continue;
    }
    atomicAdd(&deg[i], 1);
    atomicAdd(&deg[j], 1);
  }
}

__global__ void csr_fill(const int64_t* __restrict__ pairs, int64_t npairs, int64_t* __restrict__ cursor,
                         uint32_t* __restrict__ entries) {
  for (int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; p < npairs;
       p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t i = pairs[2 * p], j = pairs[2 * p + 1];
    unsigned long long si = atomicAdd(reinterpret_cast<unsigned long long*>(&cursor[i]), 1ull);
    entries[si] = static_cast<uint32_t>(j);
    unsigned long long sj = atomicAdd(reinterpret_cast<unsigned long long*>(&cursor[j]), 1ull);
    entries[sj] = static_cast<uint32_t>(i) | kSecond;
  }
}

struct CsrWs {
  int64_t* cursor;       // nrows + 1 (any list); run: int2 per row (sorted list)
  int32_t* deg;          // nrows
  unsigned int* second;  // nrows, right after `deg`
  unsigned int* found;   // right after `second`: one memset clears them
  char* scan;
  char* sort;
  uint32_t* slots;       // last, as many per row as the workspace has room for
};

// Slots per row: twice the mean number of second halves and eight (an interior
// row of a cloud with free faces, or in a shuffled order, has more than the
// mean), at most 128 and 4 GiB in all.
int64_t slots_wanted(int64_t npairs, int64_t nrows) {
  if (nrows <= 0 || npairs <= 0) return 0;
  const int64_t k = std::min<int64_t>((2 * npairs / nrows + 15) / 8 * 8, 128);
  return std::min(k, (int64_t(4) << 30) / (nrows * static_cast<int64_t>(sizeof(uint32_t))));
}

size_t csr_layout(int64_t nrows, CsrWs* w, void* base) {
  char* cur = static_cast<char*>(base);
  size_t used = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = cur ? cur + used : nullptr;
    used += align_up(bytes);
    return p;
  };
  CsrWs t{};
  t.cursor = reinterpret_cast<int64_t*>(take((nrows + 1) * sizeof(int64_t)));
  t.deg = reinterpret_cast<int32_t*>(take((2 * nrows + 1) * sizeof(int32_t)));
  t.second = t.deg ? reinterpret_cast<unsigned int*>(t.deg + nrows) : nullptr;
  t.found = t.second ? t.second + nrows : nullptr;
  t.scan = take(scan_scratch_bytes(nrows + 1));
  t.sort = take(segsort_scratch_bytes(nrows));
  t.slots = reinterpret_cast<uint32_t*>(cur + used);
  if (w) *w = t;
  return used;
}

int read_found(const unsigned int* found, unsigned int* host, cudaStream_t s) {
  TSPH_CUDA_CHECK(cudaMemcpyAsync(host, found, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
  TSPH_CUDA_CHECK(cudaStreamSynchronize(s));
  return (*host & kBad) ? TSPH_ERR_INDEX : TSPH_OK;
}

// Returns with *taken false, and nothing written to the outputs, when the list
// is not sorted; w.deg then holds the degrees of a small list's rows.
template <bool kWide>
int rows_of_sorted(const int64_t* pairs, int64_t npairs, int64_t nrows, int64_t* rowptr, uint32_t* entries,
                   const CsrWs& w, unsigned int per_row, bool* taken, cudaStream_t s) {
  int2* run = reinterpret_cast<int2*>(w.cursor);
  TSPH_CUDA_CHECK(cudaMemsetAsync(run, 0, nrows * sizeof(int2), s));
  const bool small = npairs <= kSmallList;
  if (small)
    TSPH_CUDA_CHECK(cudaMemsetAsync(w.deg, 0, (2 * nrows + 1) * sizeof(unsigned int), s));
  else
    TSPH_CUDA_CHECK(cudaMemsetAsync(w.second, 0, (nrows + 1) * sizeof(unsigned int), s));
  const unsigned g = static_cast<unsigned>((npairs + kBlock - 1) / kBlock);
  const unsigned gp = static_cast<unsigned>((npairs + kPairs * kBlock - 1) / (kPairs * kBlock));
  const auto place = small ? list_place<kWide, true> : list_place<kWide, false>;
  place<<<gp, kBlock, 0, s>>>(pairs, npairs, nrows, run, w.deg, w.second, w.slots, per_row, w.found);
  TSPH_LAUNCH_CHECK();
  unsigned int found = 0;
  int rc = read_found(w.found, &found, s);
  if (rc) return rc;
  *taken = !(found & kUnsorted);
  if (!*taken) return TSPH_OK;
  list_rows<<<static_cast<unsigned>((nrows + kBlock - 1) / kBlock), kBlock, 0, s>>>(run, w.second, nrows, w.deg);
  TSPH_LAUNCH_CHECK();
  rc = exclusive_scan_i32_to_i64(w.deg, rowptr, nrows, rowptr + nrows, w.scan, s);
  if (rc) return rc;
  if (found & kOver) {
    unsigned int* placed = reinterpret_cast<unsigned int*>(w.deg);
    TSPH_CUDA_CHECK(cudaMemsetAsync(placed, 0, nrows * sizeof(unsigned int), s));
    list_rest<kWide><<<g, kBlock, 0, s>>>(pairs, npairs, run, rowptr, w.second, per_row, placed, entries);
    TSPH_LAUNCH_CHECK();
  }
  return sort_rows(SecondHalves<kWide>{entries, rowptr, run, w.second, w.slots, per_row, pairs}, nrows,
                   found & kOver ? npairs : per_row, AsEntries{entries}, w.sort, s);
}

}  // namespace
}  // namespace tsph

using namespace tsph;

extern "C" {

int64_t tsph_csr_workspace_bytes(int64_t, int64_t nrows) {
  return static_cast<int64_t>(csr_layout(nrows, nullptr, nullptr));
}

int64_t tsph_csr_slot_bytes(int64_t npairs, int64_t nrows) {
  return nrows * slots_wanted(npairs, nrows) * static_cast<int64_t>(sizeof(uint32_t));
}

int tsph_csr_from_pairs(const int64_t* pairs, int64_t npairs, int64_t nrows, int64_t* rowptr,
                        uint32_t* entries, void* ws, int64_t ws_bytes, tsph_stream stream) {
  if (nrows < 0 || npairs < 0 || nrows >= (int64_t(1) << 31)) return TSPH_ERR_ARG;
  if (ws_bytes < tsph_csr_workspace_bytes(npairs, nrows)) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  CsrWs w;
  csr_layout(nrows, &w, ws);
  if (nrows == 0 || npairs == 0) {
    TSPH_CUDA_CHECK(cudaMemsetAsync(rowptr, 0, (nrows + 1) * sizeof(int64_t), s));
    return TSPH_OK;
  }
  const bool checked = npairs < (int64_t(1) << 31);  // by list_place
  if (checked) {
    bool taken = false;
    const bool wide = reinterpret_cast<uintptr_t>(pairs) % 16 == 0;
    const int64_t room = (ws_bytes - tsph_csr_workspace_bytes(npairs, nrows)) /
                         (nrows * static_cast<int64_t>(sizeof(uint32_t)));
    const unsigned int per_row = static_cast<unsigned int>(std::min(room, slots_wanted(npairs, nrows)));
    int rc = wide ? rows_of_sorted<true>(pairs, npairs, nrows, rowptr, entries, w, per_row, &taken, s)
                  : rows_of_sorted<false>(pairs, npairs, nrows, rowptr, entries, w, per_row, &taken, s);
    if (rc || taken) return rc;
  }
  int rc = TSPH_OK;
  if (npairs > kSmallList) {
    TSPH_CUDA_CHECK(cudaMemsetAsync(w.deg, 0, (2 * nrows + 1) * sizeof(int32_t), s));
    csr_degree<<<grid_for(npairs, 256), 256, 0, s>>>(pairs, npairs, nrows, w.deg, w.found);
    TSPH_LAUNCH_CHECK();
    unsigned int found = 0;
    if (!checked && (rc = read_found(w.found, &found, s))) return rc;
  }
  rc = exclusive_scan_i32_to_i64(w.deg, rowptr, nrows, rowptr + nrows, w.scan, s);
  if (rc) return rc;
  TSPH_CUDA_CHECK(cudaMemcpyAsync(w.cursor, rowptr, nrows * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
  csr_fill<<<grid_for(npairs, 256), 256, 0, s>>>(pairs, npairs, w.cursor, entries);
  TSPH_LAUNCH_CHECK();
  return segmented_sort_u32(entries, rowptr, nrows, 2 * npairs, w.sort, s);
}

}  // extern "C"
