// Device-wide scans, the stable LSD radix sort and the segmented row sort.
#include "common.cuh"
#include "rowsort.cuh"

namespace tsph {

// ------------------------------------------------------------------- scan ---

constexpr int kScanBlock = 512;
constexpr int kScanItems = 4;
constexpr int64_t kScanTile = kScanBlock * kScanItems;

template <class TIn>
__global__ void scan_tile_totals(const TIn* __restrict__ in, int64_t n, int64_t* __restrict__ totals,
                                 const int* __restrict__ enable) {
  if (enable && !*enable) return;
  const int64_t base = blockIdx.x * kScanTile;
  int64_t local = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int64_t i = base + threadIdx.x * kScanItems + k;
    if (i < n) local += static_cast<int64_t>(in[i]);
  }
  int64_t tot;
  block_exclusive_scan<int64_t>(local, &tot);
  if (threadIdx.x == 0) totals[blockIdx.x] = tot;
}

// kSum: `offsets` holds the tile totals and every block adds up the ones before
// it itself (at most kScanDirect of them, a few loads per thread), which saves
// the pass that scans them; otherwise it holds their exclusive scan.
template <class TIn, bool kSum>
__global__ void scan_tile_apply(const TIn* __restrict__ in, int64_t* __restrict__ out, int64_t n,
                                const int64_t* __restrict__ offsets, int64_t* __restrict__ grand,
                                const int* __restrict__ enable) {
  if (enable && !*enable) return;
  const int64_t base = blockIdx.x * kScanTile;
  int64_t vals[kScanItems];
  int64_t local = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int64_t i = base + threadIdx.x * kScanItems + k;
    vals[k] = i < n ? static_cast<int64_t>(in[i]) : 0;
    local += vals[k];
  }
  int64_t before = 0;
  if (kSum) {
    int64_t part = 0;
    for (int t = threadIdx.x; t < static_cast<int>(blockIdx.x); t += blockDim.x) part += offsets[t];
    block_exclusive_scan<int64_t>(part, &before);
  } else if (offsets) {
    before = offsets[blockIdx.x];
  }
  int64_t tot;
  int64_t run = block_exclusive_scan<int64_t>(local, &tot) + before;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int64_t i = base + threadIdx.x * kScanItems + k;
    if (i < n) out[i] = run;
    run += vals[k];
  }
  if (grand && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *grand = run;
}

// Tiles up to which a block adds up the totals before it (4 per thread):
// 4.2 M elements.  Two kernels then make a scan instead of three; at 480 k
// elements 11.5 -> 8.4 us of device time and one launch fewer.
constexpr int64_t kScanDirect = 2048;

size_t scan_scratch_bytes(int64_t n) {
  size_t bytes = 0;
  int64_t m = n;
  while (m > kScanTile) {
    m = (m + kScanTile - 1) / kScanTile;
    bytes += align_up((m + 1) * sizeof(int64_t)) * 2;
  }
  return bytes + 256;
}

template <class TIn>
static int scan_impl(const TIn* in, int64_t* out, int64_t n, int64_t* total, char* scratch,
                     cudaStream_t s, const int* enable) {
  if (n <= 0) {
    if (total) TSPH_CUDA_CHECK(cudaMemsetAsync(total, 0, sizeof(int64_t), s));
    return TSPH_OK;
  }
  const int64_t blocks = (n + kScanTile - 1) / kScanTile;
  if (blocks == 1) {
    scan_tile_apply<TIn, false><<<1, kScanBlock, 0, s>>>(in, out, n, nullptr, total, enable);
    TSPH_LAUNCH_CHECK();
    return TSPH_OK;
  }
  int64_t* totals = reinterpret_cast<int64_t*>(scratch);
  int64_t* offsets = reinterpret_cast<int64_t*>(scratch + align_up((blocks + 1) * sizeof(int64_t)));
  char* next = scratch + 2 * align_up((blocks + 1) * sizeof(int64_t));
  scan_tile_totals<TIn><<<static_cast<unsigned>(blocks), kScanBlock, 0, s>>>(in, n, totals, enable);
  TSPH_LAUNCH_CHECK();
  if (blocks <= kScanDirect) {
    scan_tile_apply<TIn, true><<<static_cast<unsigned>(blocks), kScanBlock, 0, s>>>(in, out, n, totals, total,
                                                                                    enable);
    TSPH_LAUNCH_CHECK();
    return TSPH_OK;
  }
  int rc = scan_impl<int64_t>(totals, offsets, blocks, nullptr, next, s, enable);
  if (rc) return rc;
  scan_tile_apply<TIn, false><<<static_cast<unsigned>(blocks), kScanBlock, 0, s>>>(in, out, n, offsets, total,
                                                                                   enable);
  TSPH_LAUNCH_CHECK();
  return TSPH_OK;
}

int exclusive_scan_i64(const int64_t* in, int64_t* out, int64_t n, int64_t* total, void* scratch,
                       cudaStream_t s, const int* enable) {
  return scan_impl<int64_t>(in, out, n, total, static_cast<char*>(scratch), s, enable);
}

int exclusive_scan_i32_to_i64(const int32_t* in, int64_t* out, int64_t n, int64_t* total,
                              void* scratch, cudaStream_t s, const int* enable) {
  return scan_impl<int32_t>(in, out, n, total, static_cast<char*>(scratch), s, enable);
}

// ------------------------------------------------------------- radix sort ---

constexpr int kRadixBlock = 256;
constexpr int kRadixRounds = 8;
constexpr int64_t kRadixTile = kRadixBlock * kRadixRounds;

__global__ void radix_histogram(const uint64_t* __restrict__ keys, int64_t n, int shift,
                                int32_t* __restrict__ table, int64_t nblocks, const int* __restrict__ enable) {
  if (enable && !*enable) return;
  __shared__ int32_t hist[256];
  hist[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = blockIdx.x * kRadixTile;
  for (int r = 0; r < kRadixRounds; ++r) {
    int64_t i = base + r * kRadixBlock + threadIdx.x;
    if (i < n) atomicAdd(&hist[(keys[i] >> shift) & 255u], 1);
  }
  __syncthreads();
  table[static_cast<int64_t>(threadIdx.x) * nblocks + blockIdx.x] = hist[threadIdx.x];
}

// Stable scatter: element order inside a tile is round-major, lane order
// inside a warp, warp order inside a round -- i.e. increasing global index.
__global__ void radix_scatter(const uint64_t* __restrict__ keys_in, const int32_t* __restrict__ vals_in,
                              uint64_t* __restrict__ keys_out, int32_t* __restrict__ vals_out,
                              int64_t n, int shift, const int64_t* __restrict__ offsets,
                              int64_t nblocks, const int* __restrict__ enable) {
  if (enable && !*enable) return;
  __shared__ int32_t warp_cnt[kRadixBlock / 32][256];
  __shared__ int64_t base_off[256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  base_off[threadIdx.x] = offsets[static_cast<int64_t>(threadIdx.x) * nblocks + blockIdx.x];
  const unsigned lt_mask = (1u << lane) - 1u;
  const int64_t base = blockIdx.x * kRadixTile;
  for (int r = 0; r < kRadixRounds; ++r) {
#pragma unroll
    for (int w = 0; w < kRadixBlock / 32; ++w) warp_cnt[w][threadIdx.x] = 0;
    __syncthreads();
    const int64_t i = base + r * kRadixBlock + threadIdx.x;
    const bool valid = i < n;
    uint64_t key = valid ? keys_in[i] : 0;
    int32_t val = valid ? vals_in[i] : 0;
    const unsigned digit = valid ? static_cast<unsigned>((key >> shift) & 255u) : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, digit);
    const int rank = __popc(peers & lt_mask);
    if (valid && rank == 0) warp_cnt[warp][digit] = __popc(peers);
    __syncthreads();
    // exclusive prefix over warps for digit == threadIdx.x
    {
      int32_t run = 0;
#pragma unroll
      for (int w = 0; w < kRadixBlock / 32; ++w) {
        int32_t c = warp_cnt[w][threadIdx.x];
        warp_cnt[w][threadIdx.x] = run;
        run += c;
      }
      __syncthreads();
      if (valid) {
        int64_t pos = base_off[digit] + warp_cnt[warp][digit] + rank;
        keys_out[pos] = key;
        vals_out[pos] = val;
      }
      __syncthreads();
      base_off[threadIdx.x] += run;
    }
    __syncthreads();
  }
}

size_t radix_scratch_bytes(int64_t n) {
  int64_t nblocks = (n + kRadixTile - 1) / kRadixTile;
  int64_t m = 256 * nblocks;
  return align_up(m * sizeof(int32_t)) + align_up(m * sizeof(int64_t)) + scan_scratch_bytes(m);
}

__global__ void radix_copy_back(const uint64_t* __restrict__ ks, const int32_t* __restrict__ vs,
                                uint64_t* __restrict__ kd, int32_t* __restrict__ vd, int64_t n,
                                const int* __restrict__ enable) {
  if (enable && !*enable) return;
  for (int64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    kd[i] = ks[i];
    vd[i] = vs[i];
  }
}

int radix_sort_u64_i32(uint64_t* keys, int32_t* vals, uint64_t* keys_tmp, int32_t* vals_tmp,
                       int64_t n, int bits, void* scratch, cudaStream_t s, const int* enable) {
  if (n <= 1 || bits <= 0) return TSPH_OK;
  const int64_t nblocks = (n + kRadixTile - 1) / kRadixTile;
  const int64_t m = 256 * nblocks;
  char* sc = static_cast<char*>(scratch);
  int32_t* table = reinterpret_cast<int32_t*>(sc);
  int64_t* offsets = reinterpret_cast<int64_t*>(sc + align_up(m * sizeof(int32_t)));
  char* scan_sc = sc + align_up(m * sizeof(int32_t)) + align_up(m * sizeof(int64_t));
  uint64_t *ka = keys, *kb = keys_tmp;
  int32_t *va = vals, *vb = vals_tmp;
  int passes = 0;
  for (int shift = 0; shift < bits; shift += 8, ++passes) {
    radix_histogram<<<static_cast<unsigned>(nblocks), kRadixBlock, 0, s>>>(ka, n, shift, table, nblocks,
                                                                            enable);
    TSPH_LAUNCH_CHECK();
    int rc = exclusive_scan_i32_to_i64(table, offsets, m, nullptr, scan_sc, s, enable);
    if (rc) return rc;
    radix_scatter<<<static_cast<unsigned>(nblocks), kRadixBlock, 0, s>>>(ka, va, kb, vb, n, shift,
                                                                          offsets, nblocks, enable);
    TSPH_LAUNCH_CHECK();
    uint64_t* kt = ka; ka = kb; kb = kt;
    int32_t* vt = va; va = vb; vb = vt;
  }
  if (passes & 1) {
    radix_copy_back<<<grid_for(n, 256), 256, 0, s>>>(ka, va, keys, vals, n, enable);
    TSPH_LAUNCH_CHECK();
  }
  return TSPH_OK;
}

// ---------------------------------------------------------- segmented sort ---

size_t segsort_scratch_bytes(int64_t rows) {
  return 2 * align_up(static_cast<size_t>(rows + 1) * sizeof(int64_t)) + 256;
}

int segmented_sort_u32(uint32_t* vals, const int64_t* rowptr, int64_t rows, int64_t entries, void* scratch,
                       cudaStream_t s) {
  return sort_rows(CsrRows{vals, rowptr}, rows, entries, AsEntries{vals}, scratch, s);
}

}  // namespace tsph
