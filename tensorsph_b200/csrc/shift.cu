// Lind particle shifting (particle_shifting.py:93-224) and the radix-select
// order statistic behind its reference concentration.
//
//   S1 concentration  C_a = V_a W(0) + sum_b V_b W_ab        (2-D cubic sigma,
//                     as the reference uses it in every dimension)
//   S2 gradient       grad C_a = sum_b V_b (C_b - C_a) grad_a W_ab, normal
//   Q  c_ref          95th percentile of C, linear interpolation, on device
//   S3 apply          shift = -A grad C, tangential at C < fs * c_ref, cap |shift|
#include <cmath>

#include "common.cuh"
#include "gather.cuh"
#include "sphkernels.cuh"

namespace tsph {
namespace {

// ----------------------------------------------------------- radix select ---

__device__ __forceinline__ uint64_t order_key(double v) {
  uint64_t b = static_cast<uint64_t>(__double_as_longlong(v));
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ uint32_t order_key(float v) {
  uint32_t b = __float_as_uint(v);
  return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ double from_key(uint64_t k) {
  uint64_t b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double(static_cast<long long>(b));
}
__device__ __forceinline__ double from_key(uint32_t k) {
  uint32_t b = (k >> 31) ? (k & 0x7fffffffu) : ~k;
  return static_cast<double>(__uint_as_float(b));
}

// Both ranks around the quantile, most significant digit first: per 8-bit digit
// one kernel counts the keys that share each rank's prefix, and its last block
// to finish picks the two digits (the other blocks' counts are complete by
// then; nothing waits).  4 launches for FP32 keys, 8 for FP64, against 36 with a
// kernel per step and a serial walk of the bins per rank: 200 k FP32 values in
// 20 us instead of 150.
struct SelectState {
  unsigned long long prefix[2];
  long long rank[2];
  unsigned int done;
};

__device__ __forceinline__ void select_digit(SelectState* st, int which, unsigned int* hist, int shift) {
  // one warp: prefix sums of the 256 bins, eight per lane
  const int lane = threadIdx.x & 31;
  unsigned int c[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    c[i] = *reinterpret_cast<volatile unsigned int*>(&hist[8 * lane + i]);
    sum += c[i];
  }
  const unsigned int incl = warp_inclusive_scan(sum);
  const long long k = st->rank[which];
  long long below = incl - sum;
  int digit = -1;
  long long base = 0;
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
    st->prefix[which] |= static_cast<unsigned long long>(digit) << shift;
    st->rank[which] = k - base;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) hist[8 * lane + i] = 0;
}

// torch.lerp: start + w (end - start) for w < 0.5, else end - (end - start) (1 - w)
template <class T, class K>
__global__ void __launch_bounds__(256) select_pass(const T* __restrict__ x, int64_t n, SelectState* st, int shift,
                                                   int bits_total, long long lo, long long hi, double w,
                                                   unsigned int* hist, double* out) {
  __shared__ unsigned int h[2][256];
  __shared__ bool last;
  h[0][threadIdx.x] = h[1][threadIdx.x] = 0;
  __syncthreads();
  const int hi_shift = shift + 8;
  const bool first = hi_shift >= bits_total;
  const unsigned long long p0 = first ? 0 : st->prefix[0], p1 = first ? 0 : st->prefix[1];
  const bool same = p0 == p1;
  for (int64_t a = blockIdx.x * 256ll + threadIdx.x; a < n; a += gridDim.x * 256ll) {
    const unsigned long long kk = static_cast<unsigned long long>(order_key(x[a]));
    const unsigned int digit = static_cast<unsigned int>((kk >> shift) & 255ull);
    if (first || (kk >> hi_shift) == (p0 >> hi_shift)) atomicAdd(&h[0][digit], 1u);
    if (!same && (kk >> hi_shift) == (p1 >> hi_shift)) atomicAdd(&h[1][digit], 1u);
  }
  __syncthreads();
  for (int r = 0; r < 2; ++r) {
    const unsigned int v = h[same ? 0 : r][threadIdx.x];
    if (v) atomicAdd(&hist[256 * r + threadIdx.x], v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < 2 && first) {
    st->prefix[threadIdx.x] = 0;
    st->rank[threadIdx.x] = threadIdx.x == 0 ? lo : hi;
  }
  if (threadIdx.x == 0) st->done = 0;
  __syncthreads();
  if (threadIdx.x < 64) select_digit(st, threadIdx.x >> 5, hist + 256 * (threadIdx.x >> 5), shift);
  __syncthreads();
  if (shift == 0 && threadIdx.x == 0) {
    const double u = from_key(static_cast<K>(st->prefix[0])), v = from_key(static_cast<K>(st->prefix[1]));
    *out = w < 0.5 ? u + w * (v - u) : v - (v - u) * (1.0 - w);
  }
}

template <class T>
int quantile_impl(const T* x, int64_t n, double q, double* out, char* ws, cudaStream_t s) {
  using K = typename std::conditional<sizeof(T) == 8, uint64_t, uint32_t>::type;
  const int bits = sizeof(T) * 8;
  SelectState* st = reinterpret_cast<SelectState*>(ws);
  unsigned int* hist = reinterpret_cast<unsigned int*>(ws + 256);
  TSPH_CUDA_CHECK(cudaMemsetAsync(ws, 0, 256 + 512 * sizeof(unsigned int), s));
  const double pos = q * static_cast<double>(n - 1);
  const long long lo = static_cast<long long>(std::floor(pos));
  const long long hi = static_cast<long long>(std::ceil(pos));
  const unsigned g = grid_for(n, 1024, 148 * 4);
  for (int shift = bits - 8; shift >= 0; shift -= 8) {
    select_pass<T, K><<<g, 256, 0, s>>>(x, n, st, shift, bits, lo, hi, pos - static_cast<double>(lo), hist, out);
    TSPH_LAUNCH_CHECK();
  }
  return TSPH_OK;
}

// --------------------------------------------------------------- shifting ---

template <class T, int D>
__global__ void s_pack(const T* __restrict__ pos, const T* __restrict__ vol, int64_t n, Q4<T>* __restrict__ pv) {
  for (int64_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x)
    pv[a] = Q4<T>{pos[a * D], D > 1 ? pos[a * D + 1] : T(0), D > 2 ? pos[a * D + 2] : T(0), vol[a]};
}

// C is compared with a fraction of its own 95th percentile, in the middle of
// its range, and the shift jumps where the comparison turns: in FP32, where a
// last bit of C turns it for some particle of a large cloud, C keeps one thread
// per row, the row's order and the divisions of w().  17.5 us of the 200 k
// particles' 250 either way.
template <class T, int D, int L>
__global__ void __launch_bounds__(kGatherBlock) s_concentration(int64_t n, Cubic<T> k, const Q4<T>* __restrict__ pv,
                                                                const int64_t* __restrict__ rowptr,
                                                                const uint32_t* __restrict__ ent,
                                                                T* __restrict__ c) {
  static_assert(sizeof(T) == 8 || L == 1, "FP32 rows are summed in order");
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= n) return;
  const Q4<T> pa = pv[a];
  CSum<T> s;
  if (me.lane == 0) s.add(pa.w * k.sigma);
  me.walk(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const Q4<T> pb = pv[e & kIndexMask];
    const T dx = pa.x - pb.x, dy = pa.y - pb.y, dz = pa.z - pb.z;
    const T r2 = dx * dx + dy * dy + dz * dz;
    s.add(pb.w * (sizeof(T) == 8 ? k.w2(r2) : k.w(sqrt(r2))));
  });
  const T v = me.sum(s);
  if (me.lane == 0) c[a] = v;
}

template <class T, int D, int L>
__global__ void __launch_bounds__(kGatherBlock) s_gradient(int64_t n, Cubic<T> k, const Q4<T>* __restrict__ pv,
                                                           const int64_t* __restrict__ rowptr,
                                                           const uint32_t* __restrict__ ent, const T* __restrict__ c,
                                                           T* __restrict__ grad, T* __restrict__ normal) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= n) return;
  const Q4<T> pa = pv[a];
  const T ca = c[a];
  CSum<T> g[3];
  me.walk_ahead(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const uint32_t b = e & kIndexMask;
    const Q4<T> pb = pv[b];
    const T d[3] = {pa.x - pb.x, pa.y - pb.y, pa.z - pb.z};
    const T gs = k.g2(k.radial(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]));
    const T diff = c[b] - ca;
#pragma unroll
    for (int r = 0; r < D; ++r) g[r].add(pb.w * (diff * (d[r] * gs)));
  });
  T v[3], nrm2 = T(0);
#pragma unroll
  for (int r = 0; r < D; ++r) {
    v[r] = me.sum(g[r]);
    nrm2 += v[r] * v[r];
  }
  if (me.lane) return;
  const T nrm = sqrt(nrm2);
#pragma unroll
  for (int r = 0; r < D; ++r) {
    grad[a * D + r] = v[r];
    normal[a * D + r] = nrm > T(1e-30) ? -v[r] / nrm : T(0);
  }
}

template <class T, int D>
__global__ void s_apply(int64_t n, const T* __restrict__ pos, const T* __restrict__ c,
                        const T* __restrict__ grad, const T* __restrict__ normal,
                        const double* __restrict__ c_ref_p, double free_surface, T magnitude, T cap,
                        T* __restrict__ out, T* __restrict__ shift, uint8_t* __restrict__ fs_out) {
  const double c_ref = *c_ref_p;
  const T thresh = static_cast<T>(free_surface * c_ref);
  for (int64_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
    const bool fs = c_ref > 0.0 && c[a] < thresh;
    T sh[3], nn[3];
#pragma unroll
    for (int r = 0; r < D; ++r) {
      sh[r] = -magnitude * grad[a * D + r];
      nn[r] = normal[a * D + r];
    }
    if (fs) {
      T dot = T(0);
#pragma unroll
      for (int r = 0; r < D; ++r) dot += sh[r] * nn[r];
#pragma unroll
      for (int r = 0; r < D; ++r) sh[r] = sh[r] - dot * nn[r];
    }
    T m2 = T(0);
#pragma unroll
    for (int r = 0; r < D; ++r) m2 += sh[r] * sh[r];
    const T mag = sqrt(m2);
    if (mag > cap) {
      const T sc = cap / mag;
#pragma unroll
      for (int r = 0; r < D; ++r) sh[r] = sh[r] * sc;
    }
#pragma unroll
    for (int r = 0; r < D; ++r) {
      shift[a * D + r] = sh[r];
      out[a * D + r] = pos[a * D + r] + sh[r];
    }
    if (fs_out) fs_out[a] = fs ? 1 : 0;
  }
}

__global__ void s_store_cref(double* out, double v) { *out = v; }

struct SLayout {
  size_t pv, select, total;
};

SLayout s_layout(const tsph_shift_params& p) {
  const size_t ts = p.dtype == TSPH_F64 ? 8 : 4;
  SLayout L{};
  L.pv = 0;
  L.select = align_up(p.n * 4 * ts);
  L.total = L.select + 4096;
  return L;
}

template <class T, int D>
int run_shift(const tsph_shift_params& prm, const tsph_shift_io& io, char* ws, cudaStream_t s) {
  SLayout L = s_layout(prm);
  Q4<T>* pv = reinterpret_cast<Q4<T>*>(ws + L.pv);
  const int64_t n = prm.n;
  const Cubic<T> k = make_cubic<T>(prm.h, prm.sigma);
  s_pack<T, D><<<grid_for(n, 256), 256, 0, s>>>(static_cast<const T*>(io.pos), static_cast<const T*>(io.volume),
                                                n, pv);
  with_lanes<D>(n, [&](auto lanes) -> int {
    constexpr int LN = decltype(lanes)::value;
    const unsigned g = row_grid(n, LN);
    constexpr int LC = sizeof(T) == 8 ? LN : 1;
    s_concentration<T, D, LC><<<row_grid(n, LC), kGatherBlock, 0, s>>>(n, k, pv, io.rowptr, io.entries,
                                                                       static_cast<T*>(io.concentration));
    s_gradient<T, D, LN><<<g, kGatherBlock, 0, s>>>(n, k, pv, io.rowptr, io.entries,
                                                    static_cast<const T*>(io.concentration),
                                                    static_cast<T*>(io.grad), static_cast<T*>(io.normal));
    return TSPH_OK;
  });
  TSPH_LAUNCH_CHECK();
  if (prm.c_reference < 0) {
    int rc = quantile_impl<T>(static_cast<const T*>(io.concentration), n, 0.95, io.c_reference,
                              ws + L.select, s);
    if (rc) return rc;
  } else {
    s_store_cref<<<1, 1, 0, s>>>(io.c_reference, prm.c_reference);
  }
  s_apply<T, D><<<grid_for(n, 256), 256, 0, s>>>(
      n, static_cast<const T*>(io.pos), static_cast<const T*>(io.concentration), static_cast<const T*>(io.grad),
      static_cast<const T*>(io.normal), io.c_reference, prm.free_surface, static_cast<T>(prm.magnitude),
      static_cast<T>(prm.cap), static_cast<T*>(io.out_pos), static_cast<T*>(io.shift), io.free_surface);
  TSPH_LAUNCH_CHECK();
  return TSPH_OK;
}

}  // namespace
}  // namespace tsph

using namespace tsph;

extern "C" {

int64_t tsph_quantile_workspace_bytes(int64_t n) {
  (void)n;
  return 4096;
}

int tsph_quantile(const void* x, int64_t n, int64_t dtype, double q, double* out, void* ws,
                  int64_t ws_bytes, tsph_stream stream) {
  if (n <= 0 || !(q >= 0.0 && q <= 1.0)) return TSPH_ERR_ARG;
  if (ws_bytes < tsph_quantile_workspace_bytes(n)) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == TSPH_F32) return quantile_impl<float>(static_cast<const float*>(x), n, q, out, static_cast<char*>(ws), s);
  if (dtype == TSPH_F64) return quantile_impl<double>(static_cast<const double*>(x), n, q, out, static_cast<char*>(ws), s);
  return TSPH_ERR_ARG;
}

int64_t tsph_shift_workspace_bytes(const tsph_shift_params* prm) {
  if (!prm) return -1;
  return static_cast<int64_t>(s_layout(*prm).total);
}

int tsph_shift_positions(const tsph_shift_params* prm, const tsph_shift_io* io, void* ws,
                         int64_t ws_bytes, tsph_stream stream) {
  if (!prm || !io || prm->dim < 1 || prm->dim > 3 || prm->n < 0) return TSPH_ERR_ARG;
  if (ws_bytes < tsph_shift_workspace_bytes(prm)) return TSPH_ERR_WORKSPACE;
  if (prm->n == 0) return TSPH_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  char* w = static_cast<char*>(ws);
  auto go = [&](auto t) {
    using T = decltype(t);
    if (prm->dim == 1) return run_shift<T, 1>(*prm, *io, w, s);
    if (prm->dim == 2) return run_shift<T, 2>(*prm, *io, w, s);
    return run_shift<T, 3>(*prm, *io, w, s);
  };
  if (prm->dtype == TSPH_F32) return go(float{});
  if (prm->dtype == TSPH_F64) return go(double{});
  return TSPH_ERR_ARG;
}

}  // extern "C"
