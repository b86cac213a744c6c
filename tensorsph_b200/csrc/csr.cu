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
//   order, so only the second halves need counting, scattering and sorting:
//     A  list_degrees  run boundaries, one atomic per pair that also hands out
//                      the pair's slot in row j (kept in 16 bits)
//     scan of the degrees
//     B  list_fill     the first half copied in place (coalesced), the second
//                      scattered to its slots
//     C  rows_sort     the second halves only
//   any other list: two atomics per pair to count, two to fill, rows sorted whole.
//
// What bounds the first route: the L2 atomics of A (one per pair), the
// scattered 4-byte stores of B, instruction issue in C.  18.6 M pairs of a
// periodic column (480 k rows): A 0.13, scan 0.01, B 0.15, C 0.11 ms, against
// 0.22 + 0.01 + 0.36 + 0.60 ms by the second route with a rank sort of whole
// rows; 10.6 M pairs of a 2-D column (1.04 M rows): 0.26 against 0.53 ms.
#include "common.cuh"
#include "rowsort.cuh"

namespace tsph {
namespace {

constexpr uint32_t kSecond = 0x80000000u;
constexpr int kBlock = 256;
// One pair per thread: the loads of a warp are one contiguous 512-byte run.

enum { kBad = 1, kUnsorted = 2, kLongRow = 4 };

// kWide: the list starts on a 16-byte boundary (one load per pair).
template <bool kWide>
__device__ __forceinline__ longlong2 ld_pair(const int64_t* __restrict__ pairs, int64_t p) {
  if (kWide) return *reinterpret_cast<const longlong2*>(pairs + 2 * p);
  return make_longlong2(pairs[2 * p], pairs[2 * p + 1]);
}

// A: with `found` already raised by an earlier block the rest of the grid
// returns at once (an unsorted list is seen within its first pairs).  The read
// goes through the L1, so a block may still miss the flag; it is no more than a
// short cut, and the host reads the flag after the kernel.
template <bool kWide>
__global__ void __launch_bounds__(kBlock) list_degrees(const int64_t* __restrict__ pairs, int64_t npairs,
                                                       int64_t nrows, int2* __restrict__ run,
                                                       unsigned int* __restrict__ second,
                                                       uint16_t* __restrict__ slot, unsigned int* found) {
  if (*found & kUnsorted) return;
  const int64_t p = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (p >= npairs) return;
  const longlong2 me = ld_pair<kWide>(pairs, p);
  const int64_t i = me.x, j = me.y;
  if (i < 0 || j < 0 || i >= nrows || j >= nrows) {
    atomicOr(found, kBad);
    return;
  }
  const longlong2 prev = p > 0 ? ld_pair<kWide>(pairs, p - 1) : make_longlong2(-1, -1);
  if (prev.x > i || (prev.x == i && prev.y > j)) {
    atomicOr(found, kUnsorted);
    return;
  }
  if (prev.x != i) {
    run[i].x = static_cast<int>(p);
    if (prev.x >= 0 && prev.x < nrows) run[prev.x].y = static_cast<int>(p);
  }
  if (p == npairs - 1) run[i].y = static_cast<int>(npairs);
  const unsigned int s = atomicAdd(&second[j], 1u);
  if (s > 0xffffu) atomicOr(found, kLongRow);
  slot[p] = static_cast<uint16_t>(s);
}

__global__ void list_rows(const int2* __restrict__ run, const unsigned int* __restrict__ second, int64_t nrows,
                          int32_t* __restrict__ deg) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r < nrows) deg[r] = run[r].y - run[r].x + static_cast<int32_t>(second[r]);
}

// B
template <bool kWide>
__global__ void __launch_bounds__(kBlock) list_fill(const int64_t* __restrict__ pairs, int64_t npairs,
                                                    const int2* __restrict__ run, const int64_t* __restrict__ rowptr,
                                                    const uint16_t* __restrict__ slot,
                                                    uint32_t* __restrict__ entries) {
  const int64_t p = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x;
  if (p >= npairs) return;
  const longlong2 me = ld_pair<kWide>(pairs, p);
  entries[rowptr[me.x] + (p - run[me.x].x)] = static_cast<uint32_t>(me.y);
  const int2 rj = run[me.y];
  entries[rowptr[me.y] + (rj.y - rj.x) + slot[p]] = static_cast<uint32_t>(me.x) | kSecond;
}

// The second-element halves of the rows.
struct SecondHalves {
  uint32_t* entries;
  const int64_t* rowptr;
  const int2* run;
  __device__ __forceinline__ int64_t dst(int64_t r) const { return rowptr[r] + (run[r].y - run[r].x); }
  __device__ __forceinline__ uint32_t* src(int64_t r) const { return entries + dst(r); }
  __device__ __forceinline__ int64_t len(int64_t r) const { return rowptr[r + 1] - dst(r); }
};

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
  int32_t* deg;          // nrows
  int64_t* cursor;       // nrows + 1 (any list); run: int2 per row (sorted list)
  unsigned int* second;  // nrows
  unsigned int* found;   // right after `second`: one memset clears both
  uint16_t* slot;        // npairs
  char* scan;
  char* sort;
};

size_t csr_layout(int64_t npairs, int64_t nrows, CsrWs* w, void* base) {
  char* cur = static_cast<char*>(base);
  size_t used = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = cur ? cur + used : nullptr;
    used += align_up(bytes);
    return p;
  };
  CsrWs t{};
  t.deg = reinterpret_cast<int32_t*>(take(nrows * sizeof(int32_t)));
  t.cursor = reinterpret_cast<int64_t*>(take((nrows + 1) * sizeof(int64_t)));
  t.second = reinterpret_cast<unsigned int*>(take((nrows + 1) * sizeof(unsigned int)));
  t.found = t.second ? t.second + nrows : nullptr;
  t.slot = reinterpret_cast<uint16_t*>(take(npairs * sizeof(uint16_t)));
  t.scan = take(scan_scratch_bytes(nrows + 1));
  t.sort = take(segsort_scratch_bytes(nrows));
  if (w) *w = t;
  return used;
}

int read_found(const unsigned int* found, unsigned int* host, cudaStream_t s) {
  TSPH_CUDA_CHECK(cudaMemcpyAsync(host, found, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
  TSPH_CUDA_CHECK(cudaStreamSynchronize(s));
  return (*host & kBad) ? TSPH_ERR_INDEX : TSPH_OK;
}

// Returns with *taken false, and nothing written to the outputs, when the list
// is not sorted (or a row has more than 65,536 second-element entries).
template <bool kWide>
int rows_of_sorted(const int64_t* pairs, int64_t npairs, int64_t nrows, int64_t* rowptr, uint32_t* entries,
                   const CsrWs& w, bool* taken, cudaStream_t s) {
  int2* run = reinterpret_cast<int2*>(w.cursor);
  TSPH_CUDA_CHECK(cudaMemsetAsync(run, 0, nrows * sizeof(int2), s));
  TSPH_CUDA_CHECK(cudaMemsetAsync(w.second, 0, (nrows + 1) * sizeof(unsigned int), s));
  const unsigned g = static_cast<unsigned>((npairs + kBlock - 1) / kBlock);
  list_degrees<kWide><<<g, kBlock, 0, s>>>(pairs, npairs, nrows, run, w.second, w.slot, w.found);
  TSPH_LAUNCH_CHECK();
  unsigned int found = 0;
  int rc = read_found(w.found, &found, s);
  *taken = rc != TSPH_OK || found == 0;
  // an index out of range behind an unsorted stretch is found by the general route
  if (found & kUnsorted) *taken = false;
  if (!*taken) return TSPH_OK;
  if (rc) return rc;
  list_rows<<<static_cast<unsigned>((nrows + kBlock - 1) / kBlock), kBlock, 0, s>>>(run, w.second, nrows, w.deg);
  TSPH_LAUNCH_CHECK();
  rc = exclusive_scan_i32_to_i64(w.deg, rowptr, nrows, rowptr + nrows, w.scan, s);
  if (rc) return rc;
  list_fill<kWide><<<g, kBlock, 0, s>>>(pairs, npairs, run, rowptr, w.slot, entries);
  TSPH_LAUNCH_CHECK();
  return sort_rows(SecondHalves{entries, rowptr, run}, nrows, npairs, AsEntries{entries}, w.sort, s);
}

}  // namespace
}  // namespace tsph

using namespace tsph;

extern "C" {

int64_t tsph_csr_workspace_bytes(int64_t npairs, int64_t nrows) {
  return static_cast<int64_t>(csr_layout(npairs, nrows, nullptr, nullptr));
}

int tsph_csr_from_pairs(const int64_t* pairs, int64_t npairs, int64_t nrows, int64_t* rowptr,
                        uint32_t* entries, void* ws, int64_t ws_bytes, tsph_stream stream) {
  if (nrows < 0 || npairs < 0 || nrows >= (int64_t(1) << 31)) return TSPH_ERR_ARG;
  if (ws_bytes < tsph_csr_workspace_bytes(npairs, nrows)) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  CsrWs w;
  csr_layout(npairs, nrows, &w, ws);
  if (nrows == 0 || npairs == 0) {
    TSPH_CUDA_CHECK(cudaMemsetAsync(rowptr, 0, (nrows + 1) * sizeof(int64_t), s));
    return TSPH_OK;
  }
  if (npairs < (int64_t(1) << 31)) {
    bool taken = false;
    const bool wide = reinterpret_cast<uintptr_t>(pairs) % 16 == 0;
    int rc = wide ? rows_of_sorted<true>(pairs, npairs, nrows, rowptr, entries, w, &taken, s)
                  : rows_of_sorted<false>(pairs, npairs, nrows, rowptr, entries, w, &taken, s);
    if (rc || taken) return rc;
  }
  TSPH_CUDA_CHECK(cudaMemsetAsync(w.deg, 0, nrows * sizeof(int32_t), s));
  TSPH_CUDA_CHECK(cudaMemsetAsync(w.found, 0, sizeof(unsigned int), s));
  csr_degree<<<grid_for(npairs, 256), 256, 0, s>>>(pairs, npairs, nrows, w.deg, w.found);
  TSPH_LAUNCH_CHECK();
  unsigned int found = 0;
  int rc = read_found(w.found, &found, s);
  if (rc) return rc;
  rc = exclusive_scan_i32_to_i64(w.deg, rowptr, nrows, rowptr + nrows, w.scan, s);
  if (rc) return rc;
  TSPH_CUDA_CHECK(cudaMemcpyAsync(w.cursor, rowptr, nrows * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
  csr_fill<<<grid_for(npairs, 256), 256, 0, s>>>(pairs, npairs, w.cursor, entries);
  TSPH_LAUNCH_CHECK();
  return segmented_sort_u32(entries, rowptr, nrows, 2 * npairs, w.sort, s);
}

}  // extern "C"
