// Radix select of the k-th smallest of n 64-bit keys (IEEE bits of
// non-negative floats order as unsigned integers), 8 bits a pass from bit
// `top`.  A pass is one kernel: block histograms in shared memory, one global
// add per bin, and the last block to finish picks the digit (nothing waits).
// sel[0] holds the key prefix, sel[1] the rank within it; the final key is
// sel[0].  Half the launches of a histogram and a pick kernel per pass: 482 k
// keys in 47 us against 64.  Used by kernels inside anonymous namespaces, so
// every file that includes it gets its own copy.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "common.cuh"

namespace tsph {
namespace {

// One warp: prefix sums of the 256 bins (8 per lane) find the digit.
__device__ __forceinline__ void c_pick(int shift, unsigned long long* sel, unsigned int* hist) {
  const int lane = threadIdx.x & 31;
  unsigned int c[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    c[i] = *reinterpret_cast<volatile unsigned int*>(&hist[8 * lane + i]);
    sum += c[i];
  }
  unsigned int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const unsigned long long k = sel[1];
  unsigned long long below = incl - sum;
  int digit = -1;
  unsigned long long base = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (digit < 0 && k >= below && k < below + c[i]) {
      digit = 8 * lane + i;
      base = below;
    }
    below += c[i];
  }
  __syncwarp();
  if (digit >= 0) {
    sel[0] |= static_cast<unsigned long long>(digit) << shift;
    sel[1] = k - base;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) hist[8 * lane + i] = 0;
}

// hist[256] counts the blocks that have finished.
__global__ void __launch_bounds__(256) c_select(const uint64_t* __restrict__ keys, int64_t n, int shift, int top,
                                                unsigned long long rank, unsigned long long* sel,
                                                unsigned int* hist) {
  __shared__ unsigned int h[256];
  __shared__ bool last;
  h[threadIdx.x] = 0;
  __syncthreads();
  const int hs = shift + 8;
  const bool first = hs >= top;  // the first pass counts every key
  const unsigned long long prefix = first ? 0 : sel[0];
  for (int64_t a = blockIdx.x * 256ll + threadIdx.x; a < n; a += gridDim.x * 256ll) {
    const uint64_t k = keys[a];
    if (first || (k >> hs) == (prefix >> hs)) atomicAdd(&h[(k >> shift) & 255u], 1u);
  }
  __syncthreads();
  if (h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], h[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&hist[256], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    hist[256] = 0;
    if (first) {
      sel[0] = 0;
      sel[1] = rank;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) c_pick(shift, sel, hist);
}

constexpr size_t kSelectHist = 257 * sizeof(unsigned int);

// Enqueue the whole select (top / 8 passes) of rank `rank` of keys[0, n);
// hist holds kSelectHist bytes.
inline int radix_select_u64(const uint64_t* keys, int64_t n, int top, long long rank, unsigned long long* sel,
                            unsigned int* hist, cudaStream_t s) {
  if (cudaMemsetAsync(hist, 0, kSelectHist, s) != cudaSuccess) return TSPH_ERR_CUDA;
  const unsigned grid = grid_for(n, 1024, 148 * 4);
  for (int shift = top - 8; shift >= 0; shift -= 8)
    c_select<<<grid, 256, 0, s>>>(keys, n, shift, top, static_cast<unsigned long long>(rank), sel, hist);
  return cudaGetLastError() == cudaSuccess ? TSPH_OK : TSPH_ERR_CUDA;
}

}  // namespace
}  // namespace tsph
