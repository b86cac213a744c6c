// Linked-cell neighbour search: cell keys, counting sort by cell and the exact
// pair emission of neighbor_search.py:44-120 / threed/neighbors3.py:71-142.
//
// Bit-exactness with the reference rests on three arithmetic rules, all
// applied with explicit round-to-nearest intrinsics (no FMA contraction):
//   cell    = floor(x / cutoff)            IEEE division in the dtype
//   d^2     = ((dx*dx) + dy*dy) + dz*dz    sequential, in the dtype
//   accept  = d^2 <= (dtype)(cutoff^2)
// and, for cell_order, on the order being a stable sort by row-major key.
//
// Passes (dense grids):
//   bounds -> [host: grid]
//   cell_count   key of every particle, its slot in its cell by an atomic
//   scan         first sorted position of every cell
//   cell_scatter a 16-byte record (x, y, z in FP32 from the grid's corner, in
//                cutoffs, and id) per particle, cell by cell
//   scan_rows    per particle (in cell order) the neighbours among the
//                candidates of its 3^D cells, into a fixed number of slots
//   scan -> [host: list length]
//   rows_sort    each row in index order, written out as pairs or gather rows
// Where a row outgrows its slots, or the workspace has none, a second scan_rows
// writes the rows to their places in the list before the sort.
// A grid with far more cells than particles sorts its keys instead (radix) and
// finds the cells by bisection.  The order inside a cell is arbitrary (slots
// come from atomics) and does not show: rows are sorted by index.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "fpmath.cuh"
#include "rowsort.cuh"

namespace tsph {

namespace {

constexpr int kMaxDim = 3;
constexpr int kBlock = 256;

struct GridDev {
  int dim, periodic, dense;
  int64_t ncell[kMaxDim];
  int64_t stride[kMaxDim];
  int64_t origin[kMaxDim];
  double cutoff, box[kMaxDim], width[kMaxDim];
  double scale;          // records = lengths * scale: 1 / cutoff, or 0 (band_of)
  float edge[kMaxDim];   // periodic box edges in records
};

// What the last count left in the slots: rows of this limit (kAllForward: the
// list's), this many slots each (0: none), the longest row if some row has more.
struct alignas(16) RowState {
  int longest, slots;
  long long limit;
};
constexpr long long kAllForward = -1;

__device__ __forceinline__ bool in_slots(const RowState* state, int slots, long long limit) {
  const int4 v = *reinterpret_cast<const int4*>(state);
  const uint64_t counted = static_cast<uint64_t>(static_cast<uint32_t>(v.w)) << 32 | static_cast<uint32_t>(v.z);
  return slots > 0 && v.y == slots && v.x <= slots && static_cast<long long>(counted) == limit;
}

struct BuildWs {
  uint64_t* keys;      // n (radix), or the key and slot of every particle (dense)
  uint64_t* keys_tmp;  // n
  int32_t* order;      // n, sorted: the particle (dense: in 3-D)
  int32_t* order_tmp;  // n
  float* rec;          // n, sorted: position from the grid's corner, in cutoffs (rec_at)
  int32_t* cell;       // n * dim, sorted: cell coordinates relative to origin
  int32_t* counts;     // total_cells (dense) or 1, then
  RowState* state;     // 1
  int64_t* start;      // total_cells + 1 (dense) or 1: first sorted position of a cell
  int64_t* rowptr;     // n + 1 (pair rows)
  int32_t* rowcount;   // n
  char* radix_scratch;
  char* scan_scratch;
  char* sort_scratch;
  uint32_t* slots;     // last: n * row_slots, where the workspace has room for them
};

// Slots per row: a 3-D row of 2h + 0.25 h holds 104 neighbours, half of them
// forward in lattice order and up to all in an arbitrary one; 27 in 2-D.
constexpr int kSlots[4] = {0, 16, 48, 128};
constexpr int64_t kSlotBytes = int64_t(4) << 30;  // a grid that would take more keeps none

// What a row holds: kForward b > a (the list's pairs (a, b)); kBoth every
// neighbour whose pair's first index is below the limit, as gather-row entries
// (b, with the top bit when a is the pair's second element).
enum RowKind { kForward, kBoth };

// Slots worth having: none where the mean row of a full grid already comes near
// them (most rows would be scanned twice and written twice).
int64_t wanted_slots(const tsph_grid& g, RowKind kind) {
  const int64_t k = kSlots[g.dim];
  const double ball[4] = {0.0, 2.0, 3.1416, 4.1888};
  const double mean = ball[g.dim] * static_cast<double>(g.n) / static_cast<double>(g.total_cells) *
                      (kind == kForward ? 0.5 : 1.0);
  return g.n * k * static_cast<int64_t>(sizeof(uint32_t)) <= kSlotBytes && static_cast<double>(k) > 1.2 * mean ? k : 0;
}

// Slots that a workspace of ws_bytes has room for.
int row_slots(const tsph_grid& g, RowKind kind, int64_t ws_bytes) {
  const int64_t k = wanted_slots(g, kind);
  return ws_bytes - g.workspace_bytes >= g.n * k * static_cast<int64_t>(sizeof(uint32_t)) ? static_cast<int>(k) : 0;
}

size_t build_layout(const tsph_grid& g, BuildWs* w, void* base) {
  const int64_t n = g.n;
  char* cur = static_cast<char*>(base);
  size_t used = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = cur ? cur + used : nullptr;
    used += align_up(bytes);
    return p;
  };
  const int64_t cells = g.dense ? g.total_cells : 1;
  BuildWs t{};
  t.keys = reinterpret_cast<uint64_t*>(take(n * sizeof(uint64_t)));
  t.keys_tmp = reinterpret_cast<uint64_t*>(take(n * sizeof(uint64_t)));
  t.order = reinterpret_cast<int32_t*>(take(n * sizeof(int32_t)));
  t.order_tmp = reinterpret_cast<int32_t*>(take(n * sizeof(int32_t)));
  t.rec = reinterpret_cast<float*>(take((n + 3) / 4 * 4 * sizeof(float4)));
  t.cell = reinterpret_cast<int32_t*>(take(n * g.dim * sizeof(int32_t)));
  t.counts = reinterpret_cast<int32_t*>(take(cells * sizeof(int32_t)));
  t.state = reinterpret_cast<RowState*>(take(sizeof(RowState)));
  t.start = reinterpret_cast<int64_t*>(take((cells + 1) * sizeof(int64_t)));
  t.rowptr = reinterpret_cast<int64_t*>(take((n + 1) * sizeof(int64_t)));
  t.rowcount = reinterpret_cast<int32_t*>(take(n * sizeof(int32_t)));
  t.radix_scratch = take(radix_scratch_bytes(n));
  t.scan_scratch = take(scan_scratch_bytes(std::max<int64_t>(n, cells) + 1));
  t.sort_scratch = take(segsort_scratch_bytes(n));
  t.slots = reinterpret_cast<uint32_t*>(cur + used);
  if (w) *w = t;
  return used;
}

// Where record t's first coordinate is and how far apart the others are.  In 3-D
// records stand in blocks of four, four x, four y, four z, so that four candidates
// are loaded 16 bytes at a time and computed two to an instruction; below, where a
// run holds a dozen candidates, one record is 16 bytes (position and particle).
template <int D>
__device__ __forceinline__ int64_t rec_at(int64_t t) {
  return D == 3 ? (t >> 2) * 12 + (t & 3) : 4 * t;
}
template <int D>
constexpr int kRecStep = D == 3 ? 4 : 1;

// Which candidates the FP32 records decide.  Records are in units of the cutoff:
// in the caller's units a squared FP32 distance overflows beyond 1.8e19 and
// vanishes below 1e-23.  A record's coordinate is within 2^-24 of the extent of
// its true value (and so is an image's shift), so a distance taken from two of
// them in FP32, and the reference's own distance in its dtype, differ by less
// than w = 2^-20 extent + 2e-6.  Below (1 - w)^2 a candidate is in, above
// (1 + w)^2 it is out; between them (about one candidate in 10^4) the
// reference's arithmetic on the given positions decides.  It decides for every
// candidate where the band would be wide (a grid of many thousand cells on an
// axis, or positions as many cutoffs outside their box), where a periodic axis
// has three cells, so that a stencil cell's image need not be the nearest one,
// and where the square of the cutoff leaves the dtype's range: the records are
// zero then, which lies between the bounds.
struct Band {
  float in, out;
  bool exact;
};

Band band_of(const tsph_grid& g) {
  const double c2 = g.cutoff * g.cutoff, far = g.dtype == TSPH_F32 ? 1e30 : 1e280;
  double extent = 0.0;
  bool exact = !(c2 > 1.0 / far && c2 < far);
  for (int k = 0; k < g.dim; ++k) {
    if (g.periodic) {
      extent = std::max(extent, std::max(g.box[k] / g.cutoff, 2.0 * static_cast<double>(g.origin[k])));
      if (g.ncell[k] < 4) exact = true;
    } else {
      extent = std::max(extent, static_cast<double>(g.ncell[k]));
    }
  }
  const double w = extent / 1048576.0 + 2e-6;
  if (exact || !(w < 0.25)) return Band{-1.f, 1.f, true};
  return Band{static_cast<float>((1.0 - w) * (1.0 - w) * (1.0 - 1e-6)),
              static_cast<float>((1.0 + w) * (1.0 + w) * (1.0 + 1e-6)), false};
}

GridDev to_dev(const tsph_grid& g) {
  GridDev d{};
  d.scale = band_of(g).exact ? 0.0 : 1.0 / g.cutoff;
  d.dim = static_cast<int>(g.dim);
  d.periodic = static_cast<int>(g.periodic);
  d.dense = static_cast<int>(g.dense);
  d.cutoff = g.cutoff;
  for (int k = 0; k < kMaxDim; ++k) {
    d.ncell[k] = k < g.dim ? g.ncell[k] : 1;
    d.origin[k] = g.origin[k];
    d.box[k] = g.box[k];
    d.width[k] = g.width[k];
    d.edge[k] = static_cast<float>(g.box[k] * d.scale);
  }
  int64_t s = 1;
  for (int k = static_cast<int>(g.dim) - 1; k >= 0; --k) {
    d.stride[k] = s;
    s *= d.ncell[k];
  }
  return d;
}

// ------------------------------------------------------------------ plan ---

template <class F>
int dispatch(int64_t dtype, int64_t dim, F&& f) {
  if (dtype == TSPH_F32) {
    if (dim == 1) return f(float{}, std::integral_constant<int, 1>{});
    if (dim == 2) return f(float{}, std::integral_constant<int, 2>{});
    if (dim == 3) return f(float{}, std::integral_constant<int, 3>{});
  } else if (dtype == TSPH_F64) {
    if (dim == 1) return f(double{}, std::integral_constant<int, 1>{});
    if (dim == 2) return f(double{}, std::integral_constant<int, 2>{});
    if (dim == 3) return f(double{}, std::integral_constant<int, 3>{});
  }
  return TSPH_ERR_ARG;
}

// out[0..2] smallest cell per axis, out[3..5] largest, out[6] 0 when some
// coordinate is not finite.  All are unsigned minima, so one memset of ones
// starts them: a cell is stored with its sign bit flipped, a largest one as
// the complement of that.  One atomic per value and block: with one per warp
// the 57 k atomics on six addresses took 43 us of 1 M FP64 particles, now 12.
template <class T, int D>
__global__ void __launch_bounds__(kBlock) bounds_kernel(const T* __restrict__ pos, int64_t n, T cutoff,
                                                        unsigned long long* __restrict__ out) {
  constexpr unsigned long long kSign = 1ull << 63;
  constexpr int kWarps = kBlock / 32;
  __shared__ unsigned long long red[kWarps][2 * D + 1];
  unsigned long long v[2 * D + 1];
#pragma unroll
  for (int k = 0; k <= 2 * D; ++k) v[k] = ~0ull;
  for (int64_t a = blockIdx.x * static_cast<int64_t>(kBlock) + threadIdx.x; a < n;
       a += static_cast<int64_t>(gridDim.x) * kBlock) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const T x = pos[a * D + k];
      if (!isfinite(x)) { v[2 * D] = 0; continue; }
      const unsigned long long c =
          static_cast<unsigned long long>(static_cast<long long>(floor(fp<T>::div(x, cutoff)))) ^ kSign;
      v[k] = c < v[k] ? c : v[k];
      v[D + k] = ~c < v[D + k] ? ~c : v[D + k];
    }
  }
#pragma unroll
  for (int k = 0; k <= 2 * D; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = w < v[k] ? w : v[k];
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = v[k];
  }
  __syncthreads();
  if (threadIdx.x <= 2 * D) {
    const int k = threadIdx.x;
    unsigned long long m = red[0][k];
    for (int w = 1; w < kWarps; ++w) m = red[w][k] < m ? red[w][k] : m;
    if (m != ~0ull) atomicMin(&out[k < D ? k : (k < 2 * D ? 3 + k - D : 6)], m);
  }
}

template <class T, int D>
int plan_bounds(const void* pos, int64_t n, double cutoff, unsigned long long* dev, cudaStream_t s) {
  TSPH_CUDA_CHECK(cudaMemsetAsync(dev, 0xff, 8 * sizeof(unsigned long long), s));
  bounds_kernel<T, D><<<grid_for(n, kBlock, 148 * 8), kBlock, 0, s>>>(
      static_cast<const T*>(pos), n, static_cast<T>(cutoff), dev);
  TSPH_LAUNCH_CHECK();
  return TSPH_OK;
}

// ----------------------------------------------------------------- build ---

__device__ __forceinline__ float record(double length, double scale) {
  return scale == 0.0 ? 0.f : static_cast<float>(length * scale);
}

// Cell of one coordinate (relative to the grid's origin, or wrapped into the
// box) and its record: the coordinate from the grid's corner, moved by whole
// boxes into the same cell when periodic, in cutoffs.
template <class T>
__device__ __forceinline__ long long cell_of(T x, const GridDev& g, int k, float* local) {
  if (g.periodic) {
    const long long raw = static_cast<long long>(floor(fp<T>::div(x, static_cast<T>(g.width[k]))));
    long long c = raw % g.ncell[k];
    if (c < 0) c += g.ncell[k];
    if (local)
      *local = record(static_cast<double>(x) - static_cast<double>((raw - c) / g.ncell[k]) *
                                                   static_cast<double>(static_cast<T>(g.box[k])), g.scale);
    return c;
  }
  if (local) *local = record(static_cast<double>(x) - static_cast<double>(g.origin[k]) * g.cutoff, g.scale);
  return static_cast<long long>(floor(fp<T>::div(x, static_cast<T>(g.cutoff)))) - g.origin[k];
}

template <class T, int D>
__device__ __forceinline__ uint64_t key_of(const T* __restrict__ pos, int64_t a, const GridDev& g, int* c, float* local) {
  uint64_t key = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const long long ck = cell_of<T>(pos[a * D + k], g, k, local ? local + k : nullptr);
    if (c) c[k] = static_cast<int>(ck);
    key += static_cast<uint64_t>(ck) * static_cast<uint64_t>(g.stride[k]);
  }
  return key;
}

template <class T, int D>
__global__ void key_kernel(const T* __restrict__ pos, int64_t n, GridDev g, uint64_t* __restrict__ keys,
                           int32_t* __restrict__ vals) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    keys[a] = key_of<T, D>(pos, a, g, nullptr, nullptr);
    vals[a] = static_cast<int32_t>(a);
  }
}

// The slot of every particle in its cell.  2 x 4 bytes a particle instead of
// the radix sort's 24 per digit, and four launches instead of five per digit.
template <class T, int D>
__global__ void cell_count(const T* __restrict__ pos, int64_t n, GridDev g, int32_t* __restrict__ counts,
                           int32_t* __restrict__ slots) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x)
    slots[a] = atomicAdd(&counts[key_of<T, D>(pos, a, g, nullptr, nullptr)], 1);
}

// Records in cell order: to start[key] + slot (dense), or from the sorted order.
template <class T, int D, bool kDense>
__global__ void cell_scatter(const T* __restrict__ pos, int64_t n, GridDev g, const int64_t* __restrict__ start,
                             const int32_t* __restrict__ slots, int32_t* __restrict__ order,
                             float* __restrict__ rec, int32_t* __restrict__ cell) {
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t a = kDense ? t : order[t];
    int c[D];
    float x[3] = {0.f, 0.f, 0.f};
    const uint64_t key = key_of<T, D>(pos, a, g, c, x);
    const int64_t at = kDense ? start[key] + slots[a] : t;
    if (D < 3) {
      reinterpret_cast<float4*>(rec)[at] = make_float4(x[0], x[1], 0.f, __int_as_float(static_cast<int>(a)));
    } else {
#pragma unroll
      for (int k = 0; k < D; ++k) rec[rec_at<D>(at) + 4 * k] = x[k];
      if (kDense) order[at] = static_cast<int>(a);
    }
#pragma unroll
    for (int k = 0; k < D; ++k) cell[at * D + k] = c[k];
  }
}

__global__ void order_to_i64(const int32_t* __restrict__ order, int64_t n, int64_t* __restrict__ out) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[a] = order[a];
}

// --------------------------------------------------------------- pairs ---

__device__ __forceinline__ int64_t lower_bound(const uint64_t* __restrict__ keys, int64_t n, uint64_t key) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (keys[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

template <class T, int D>
__device__ __forceinline__ T pair_d2(const T* __restrict__ pos, int64_t a, int64_t b, const GridDev& g) {
  T acc = T(0);
#pragma unroll
  for (int k = 0; k < D; ++k) {
    T d = fp<T>::sub(pos[a * D + k], pos[b * D + k]);
    if (g.periodic) d = fp<T>::min_image(d, static_cast<T>(g.box[k]));
    T sq = fp<T>::mul(d, d);
    acc = k == 0 ? sq : fp<T>::add(acc, sq);
  }
  return acc;
}

struct Cells {
  const float* rec;
  const int32_t* id;
  const int32_t* cell;
  const int64_t* start;   // dense
  const uint64_t* keys;   // not dense: sorted
};

// Two FP32 operations in one instruction, each rounded as its scalar form.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
// bits <- bits, sign of the low half, sign of the high half
__device__ __forceinline__ void push_signs(uint32_t& bits, uint64_t v) {
  const uint32_t lo = static_cast<uint32_t>(v), hi = static_cast<uint32_t>(v >> 32);
  bits = __funnelshift_l(hi, __funnelshift_l(lo, bits, 1), 1);
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

enum RowPass { kCount, kSlot, kFill };

// The rows of all particles, thread per row (kLanes = 1) or kLanes lanes per
// row, in cell order, so that the lanes of a warp walk the same cells.  The
// cells c - 1 .. c + 1 of the last axis are consecutive keys: a column's
// candidates are one run (two at a periodic seam), 3^(D-1) runs in all.
// kCount counts them, kSlot also writes the first `slots` of each row to its
// slots (in any order), raises state->longest where that was not all and notes
// what the slots hold; kFill, for rows that the slots do not hold, writes them
// from rowptr on, each within its own part (a rowptr of another limit would not
// fit: what is missing there becomes the row itself, so that no pass reads out of range).
//
// What bounds it: instruction issue (in 3-D three to four instructions a candidate
// and twenty a hit; the list at 2.05 h scans ~500 candidates for ~80 hits) and, with
// the stores of kSlot, scattered 4-byte writes.  1.0 M FP64 particles in 3-D: 0.48
// ms; with compares and predicates in place of the signs 0.55, and 1.55 ms to
// count and 1.65 to write with a thread per particle in the caller's order, FP64
// distances for every candidate and 27 cells by division.
template <class T, int D, RowKind kKind, RowPass kPass, int kLanes>
__global__ void __launch_bounds__(128) scan_rows(const T* __restrict__ pos, int64_t n, int64_t row_limit, GridDev g,
                                                 Cells cs, Band band, T c2, int32_t* __restrict__ rowcount,
                                                 const int64_t* __restrict__ rowptr, uint32_t* __restrict__ out,
                                                 int slots, RowState* state) {
  const long long rows_of = kKind == kForward ? kAllForward : static_cast<long long>(row_limit);
  if (kPass == kFill && in_slots(state, slots, rows_of)) return;
  constexpr int kColumns = D == 1 ? 1 : (D == 2 ? 3 : 9);
  constexpr uint32_t kSecond = 0x80000000u;
  const int lane = threadIdx.x & 31, gl = lane & (kLanes - 1);
  const unsigned group = kLanes == 1 ? 1u << lane : ((kLanes == 32 ? 0u : 1u << kLanes) - 1u) << (lane - gl);
  const int64_t t = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / kLanes;
  if (t >= n) return;
  if (kPass == kSlot && t == 0 && gl == 0) {
    state->slots = slots;
    state->limit = rows_of;
  }
  const float* ra = cs.rec + rec_at<D>(t);
  const int64_t a = D == 3 ? cs.id[t] : __float_as_int(ra[3]);
  if (kKind == kForward && kPass == kFill && a >= row_limit) return;
  int c[3] = {0, 0, 0};
#pragma unroll
  for (int k = 0; k < D; ++k) c[k] = cs.cell[t * D + k];
  const float xa[3] = {ra[0], D > 1 ? ra[kRecStep<D>] : 0.f, D > 2 ? ra[2 * kRecStep<D>] : 0.f};
  int count = 0;
  const int64_t slot = kPass == kFill ? rowptr[a] : a * slots;
  const int room = kPass == kFill ? static_cast<int>(rowptr[a + 1] - slot) : slots;

  const int me = static_cast<int>(a), limit = static_cast<int>(row_limit);
  const bool first = me < limit;  // kBoth: a row below the limit takes every neighbour
  const T* __restrict__ px = pos;
  auto put = [&](int at, int b) {
    if (at >= room) return;
    out[slot + at] = kKind == kBoth && b < me ? static_cast<uint32_t>(b) | kSecond : static_cast<uint32_t>(b);
  };
  const auto wanted = [&](int b) { return kKind == kForward ? b > me : b != me && (first || b < limit); };
  // A thread's own row, 1-D and 2-D: four candidates at once; the tests against the
  // outer bound are predicates, and one branch per batch looks at those between the
  // bounds (by signs a 2-D pass of 200 k rows takes 47 us, so 38).
  auto run_batch = [&](int beg, int end, float x, float y) {
    const float4* recs = reinterpret_cast<const float4*>(cs.rec);
    for (int p0 = beg; p0 < end; p0 += 4) {
      float4 rb[4];
      bool hit[4];
      bool unsure = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) rb[j] = recs[min(p0 + j, end - 1)];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float dx = x - rb[j].x, dy = y - rb[j].y;
        float d2 = dx * dx;
        if (D > 1) d2 = fmaf(dy, dy, d2);
        hit[j] = d2 < band.out && wanted(__float_as_int(rb[j].w)) && p0 + j < end;
        unsure |= hit[j] && d2 > band.in;
      }
      if (unsure) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (hit[j]) hit[j] = pair_d2<T, D>(px, a, __float_as_int(rb[j].w), g) <= c2;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (kPass != kCount && hit[j]) put(count, __float_as_int(rb[j].w));
        count += hit[j];
      }
    }
  };
  // A thread's own row, 3-D.  Up to 32 candidates leave the signs of d^2 - out and
  // d^2 - in in a word each (a subtraction, two to an instruction, and a shift, where
  // a compare and its predicate logic cost three on the integer pipe, which bounded
  // the pass), and of a - b; then the few that are in are looked at one by one.
  auto run_signs = [&](int beg, int end, float x, float y, float z) {
    const uint64_t xx = pack2(x, x), yy = pack2(y, y), zz = pack2(z, z);
    const uint64_t in2 = pack2(band.in, band.in), out2 = pack2(band.out, band.out);
    for (int q = beg & ~3; q < end; q += 32) {
      const ulonglong2* blk = reinterpret_cast<const ulonglong2*>(cs.rec + rec_at<3>(q));
      const int blocks = min(8, (end - q + 3) >> 2);
      uint32_t hits = 0, sure = 0, after = 0;
      const int4* ids = reinterpret_cast<const int4*>(cs.id + q);
#pragma unroll 2
      for (int i = 0; i < blocks; ++i, blk += 3) {
        const ulonglong2 bx = blk[0], by = blk[1], bz = blk[2];
        uint64_t d0 = sub2(xx, bx.x), d1 = sub2(xx, bx.y);
        const uint64_t e0 = sub2(yy, by.x), e1 = sub2(yy, by.y), f0 = sub2(zz, bz.x), f1 = sub2(zz, bz.y);
        d0 = fma2(f0, f0, fma2(e0, e0, mul2(d0, d0)));
        d1 = fma2(f1, f1, fma2(e1, e1, mul2(d1, d1)));
        push_signs(hits, sub2(d0, out2));
        push_signs(hits, sub2(d1, out2));
        push_signs(sure, sub2(d0, in2));
        push_signs(sure, sub2(d1, in2));
        if (kKind == kForward) {
          const int4 b = ids[i];
          after = __funnelshift_l(me - b.x, after, 1);
          after = __funnelshift_l(me - b.y, after, 1);
          after = __funnelshift_l(me - b.z, after, 1);
          after = __funnelshift_l(me - b.w, after, 1);
        }
      }
      if (kKind == kForward) hits &= after;
      hits <<= 32 - 4 * blocks;
      sure <<= 32 - 4 * blocks;
      // the blocks at the run's ends hold other cells' particles too
      if (q < beg) hits &= 0xffffffffu >> (beg - q);
      if (end - q < 32) hits &= ~(0xffffffffu >> (end - q));
      for (uint32_t doubt = hits & ~sure; doubt;) {
        const int k = __clz(doubt);
        doubt ^= 0x80000000u >> k;
        if (!(pair_d2<T, D>(px, a, cs.id[q + k], g) <= c2)) hits ^= 0x80000000u >> k;
      }
      while (hits) {
        const int k = __clz(hits);
        hits ^= 0x80000000u >> k;
        const int b = cs.id[q + k];
        const bool in = kKind == kForward || wanted(b);
        if (kPass != kCount && in) put(count, b);
        count += in;
      }
    }
  };
  auto run_shared = [&](int beg, int end, float x, float y, float z) {
    for (int p0 = beg; p0 < end; p0 += kLanes) {
      const int at = min(p0 + gl, end - 1);
      const float* rb = cs.rec + rec_at<D>(at);
      const int b = D == 3 ? cs.id[at] : __float_as_int(rb[3]);
      const float dx = x - rb[0];
      float d2 = dx * dx;
      if (D > 1) d2 = fmaf(y - rb[kRecStep<D>], y - rb[kRecStep<D>], d2);
      if (D > 2) d2 = fmaf(z - rb[2 * kRecStep<D>], z - rb[2 * kRecStep<D>], d2);
      bool hit = d2 < band.out && wanted(b) && p0 + gl < end;
      if (hit && d2 > band.in) hit = pair_d2<T, D>(px, a, b, g) <= c2;
      if (kPass != kCount) {
        const unsigned m = __ballot_sync(group, hit) & group;
        if (hit) put(count + __popc(m & ((1u << lane) - 1u)), b);
        count += __popc(m);
      } else {
        count += hit;
      }
    }
  };
  auto run = [&](int beg, int end, float x, float y, float z) {
    if constexpr (kLanes > 1)
      run_shared(beg, end, x, y, z);
    else if constexpr (D == 3)
      run_signs(beg, end, x, y, z);
    else
      run_batch(beg, end, x, y);
  };
  // first sorted position of cells [k0, k1] of the key space
  auto cells = [&](int64_t k0, int64_t k1, float x, float y, float z) {
    int64_t beg, end;
    if (g.dense) {
      beg = cs.start[k0];
      end = cs.start[k1 + 1];
    } else {
      beg = lower_bound(cs.keys, n, static_cast<uint64_t>(k0));
      end = lower_bound(cs.keys, n, static_cast<uint64_t>(k1) + 1);
    }
    run(static_cast<int>(beg), static_cast<int>(end), x, y, z);
  };

#pragma unroll 1
  for (int m = 0; m < kColumns; ++m) {
    const int off[2] = {m % 3 - 1, m / 3 - 1};
    float x[3] = {xa[0], xa[1], xa[2]};
    int64_t column = 0;
    bool inside = true;
#pragma unroll
    for (int k = 0; k + 1 < D; ++k) {
      int64_t nc = c[k] + off[k];
      if (g.periodic) {
        if (nc < 0) { nc += g.ncell[k]; x[k] += g.edge[k]; }
        else if (nc >= g.ncell[k]) { nc -= g.ncell[k]; x[k] -= g.edge[k]; }
      } else if (nc < 0 || nc >= g.ncell[k]) {
        inside = false;
      }
      column += nc * g.stride[k];
    }
    if (!inside) continue;
    const int64_t last = g.ncell[D - 1] - 1;
    const int64_t z0 = c[D - 1] > 0 ? c[D - 1] - 1 : 0, z1 = c[D - 1] < last ? c[D - 1] + 1 : last;
    cells(column + z0, column + z1, x[0], x[1], x[2]);
    if (g.periodic) {
      const float edge = g.edge[D - 1];
      if (c[D - 1] == 0) {
        x[D - 1] += edge;
        cells(column + last, column + last, x[0], x[1], x[2]);
        x[D - 1] -= edge;
      }
      if (c[D - 1] == last) {
        x[D - 1] -= edge;
        cells(column, column, x[0], x[1], x[2]);
      }
    }
  }
  if (kPass == kFill) {
    for (int k = count + gl; k < room; k += kLanes) out[slot + k] = static_cast<uint32_t>(me);
  } else {
    if (kPass == kCount && kLanes > 1) {
#pragma unroll
      for (int o = kLanes / 2; o > 0; o >>= 1) count += __shfl_xor_sync(group, count, o);
    }
    if (gl == 0) {
      rowcount[a] = count;
      if (kPass == kSlot && count > slots) atomicMax(&state->longest, count);
    }
  }
}

// Rows up to which eight lanes share a row: a row per thread leaves most of the
// chip idle there, eight lanes leave a sixth of theirs idle in every run.  Whole
// searches (FP32, 3-D, 2.05 h) with eight lanes / one: 8 k particles 132 / 156
// us, 20 k 137 / 144, 40 k 177 / 154, 100 k 281 / 205; 2-D: the same up to 20 k,
// 123 / 116 at 40 k.  Where every candidate takes the exact arithmetic, a thread
// looks at its candidates one by one, and eight lanes pay at any number of rows
// (FP32, three cells on two axes: 60 k rows of ~70 neighbours 366 / 488 us, of ~550
// 2.9 / 4.5 ms; on all three axes 30 k rows of ~2900 22.8 / 45.2 ms), unless the cells
// are found by bisection, which each lane would repeat (97 k rows 601 / 392 us).
constexpr int64_t kLaneRows = 24576;

template <class T, int D, RowKind kKind, RowPass kPass>
int launch_rows(const void* pos, const tsph_grid& grid, int64_t row_limit, const BuildWs& w, const int64_t* rowptr,
                uint32_t* out, int slots, cudaStream_t s) {
  const int64_t n = grid.n;
  const Cells cs{w.rec, w.order, w.cell, w.start, w.keys};
  const T c2 = static_cast<T>(grid.cutoff * grid.cutoff);
  const T* p = static_cast<const T*>(pos);
  const Band band = band_of(grid);
  if (n <= kLaneRows || (band.exact && grid.dense))
    scan_rows<T, D, kKind, kPass, 8><<<static_cast<unsigned>((n * 8 + 127) / 128), 128, 0, s>>>(
        p, n, row_limit, to_dev(grid), cs, band, c2, w.rowcount, rowptr, out, slots, w.state);
  else
    scan_rows<T, D, kKind, kPass, 1><<<static_cast<unsigned>((n + 127) / 128), 128, 0, s>>>(
        p, n, row_limit, to_dev(grid), cs, band, c2, w.rowcount, rowptr, out, slots, w.state);
  TSPH_LAUNCH_CHECK();
  return TSPH_OK;
}

// Row lengths (and the rows in their slots), scanned into rowptr.
template <RowKind kKind>
int count_rows(const void* pos, const tsph_grid& grid, int64_t row_limit, const BuildWs& w, int slots,
               int64_t* rowptr, cudaStream_t s) {
  TSPH_CUDA_CHECK(cudaMemsetAsync(w.state, 0, sizeof(RowState), s));
  int rc = dispatch(grid.dtype, grid.dim, [&](auto t, auto d) {
    using T = decltype(t);
    constexpr int D = decltype(d)::value;
    return slots ? launch_rows<T, D, kKind, kSlot>(pos, grid, row_limit, w, nullptr, w.slots, slots, s)
                 : launch_rows<T, D, kKind, kCount>(pos, grid, row_limit, w, nullptr, nullptr, 0, s);
  });
  if (rc) return rc;
  return exclusive_scan_i32_to_i64(w.rowcount, rowptr, grid.n, rowptr + grid.n, w.scan_scratch, s);
}

// The rows in their slots, or in `full` when the slots do not hold them.
struct FoundRows {
  uint32_t *slot, *full;
  const int64_t* ptr;
  const RowState* state;
  int slots;
  long long limit;
  __device__ __forceinline__ uint32_t* src(int64_t r) const {
    return in_slots(state, slots, limit) ? slot + r * slots : full + ptr[r];
  }
  __device__ __forceinline__ int64_t dst(int64_t r) const { return ptr[r]; }
  __device__ __forceinline__ int64_t len(int64_t r) const { return ptr[r + 1] - ptr[r]; }
};

// The first `rows` rows sorted into out; `full`: room for their `count` entries.
template <RowKind kKind, class Out>
int emit_rows(const void* pos, const tsph_grid& grid, int64_t row_limit, int64_t rows, const BuildWs& w, int slots,
              const int64_t* rowptr, uint32_t* full, int64_t count, Out out, cudaStream_t s) {
  int rc = dispatch(grid.dtype, grid.dim, [&](auto t, auto d) {
    return launch_rows<decltype(t), decltype(d)::value, kKind, kFill>(pos, grid, row_limit, w, rowptr, full, slots, s);
  });
  if (rc) return rc;
  const long long limit = kKind == kForward ? kAllForward : static_cast<long long>(row_limit);
  return sort_rows(FoundRows{w.slots, full, rowptr, w.state, slots, limit}, rows, count,
                   out, w.sort_scratch, s);
}

// --------------------------------------------------------- brute force ---

template <class T, int D, int MODE>
__global__ void brute_kernel(const T* __restrict__ pos, int64_t n, T c2, int32_t* __restrict__ rowcount,
                             const int64_t* __restrict__ rowptr, int64_t* __restrict__ pairs) {
  GridDev g{};
  for (int64_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
    int64_t slot = MODE == 1 ? rowptr[a] : 0;
    int32_t count = 0;
    for (int64_t b = a + 1; b < n; ++b) {
      if (pair_d2<T, D>(pos, a, b, g) <= c2) {
        if (MODE == 1) {
          pairs[2 * (slot + count)] = a;
          pairs[2 * (slot + count) + 1] = b;
        }
        ++count;
      }
    }
    if (MODE == 0) rowcount[a] = count;
  }
}

// ------------------------------------------------------- displacement ---

template <class T, int D>
__global__ void displacement_kernel(const T* __restrict__ pos, const T* __restrict__ anchor, int64_t n,
                                    int periodic, double bx, double by, double bz,
                                    unsigned long long* __restrict__ out) {
  double best = 0.0;
  const double boxv[3] = {bx, by, bz};
  for (int64_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
    T acc = T(0);
#pragma unroll
    for (int k = 0; k < D; ++k) {
      T d = fp<T>::sub(pos[a * D + k], anchor[a * D + k]);
      if (periodic) d = fp<T>::min_image(d, static_cast<T>(boxv[k]));
      acc = fp<T>::add(acc, fp<T>::mul(d, d));
    }
    double v = static_cast<double>(sqrt(acc));
    best = v > best ? v : best;
  }
  best = warp_reduce_max(best);
  if ((threadIdx.x & 31) == 0) atomicMax(out, static_cast<unsigned long long>(__double_as_longlong(best)));
}

template <class T>
T host_cutoff_sq(double cutoff) {
  return static_cast<T>(cutoff * cutoff);
}

}  // namespace

}  // namespace tsph

using namespace tsph;

extern "C" {

int64_t tsph_grid_plan_scratch_bytes(void) { return 256; }

int tsph_grid_plan(const void* pos, int64_t n, int64_t dim, int64_t dtype, double cutoff,
                   const double* box, void* scratch, tsph_grid* grid, tsph_stream stream) {
  if (!grid || dim < 1 || dim > 3 || n < 0 || (dtype != TSPH_F32 && dtype != TSPH_F64))
    return TSPH_ERR_ARG;
  if (!std::isfinite(cutoff) || cutoff <= 0) return TSPH_ERR_ARG;
  if (n > (int64_t(1) << 31) - 2) return TSPH_ERR_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  std::memset(grid, 0, sizeof(*grid));
  grid->n = n;
  grid->dim = dim;
  grid->dtype = dtype;
  grid->cutoff = cutoff;
  grid->periodic = box != nullptr;
  long long host[6] = {0, 0, 0, 0, 0, 0};
  if (n > 0) {
    unsigned long long* dev = static_cast<unsigned long long*>(scratch);
    unsigned long long raw[8];
    int rc = dispatch(dtype, dim, [&](auto t, auto d) {
      return plan_bounds<decltype(t), decltype(d)::value>(pos, n, cutoff, dev, s);
    });
    if (rc) return rc;
    TSPH_CUDA_CHECK(cudaMemcpyAsync(raw, dev, sizeof(raw), cudaMemcpyDeviceToHost, s));
    TSPH_CUDA_CHECK(cudaStreamSynchronize(s));
    if (raw[6] == 0) return TSPH_ERR_NONFINITE;
    for (int k = 0; k < dim; ++k) {
      host[k] = static_cast<long long>(raw[k] ^ (1ull << 63));
      host[3 + k] = static_cast<long long>(~raw[3 + k] ^ (1ull << 63));
    }
  }
  double cells = 1.0;
  for (int k = 0; k < 3; ++k) {
    if (k >= dim) {
      grid->ncell[k] = 1;
      continue;
    }
    if (box) {
      grid->box[k] = box[k];
      if (!(box[k] > 0) || !std::isfinite(box[k])) return TSPH_ERR_ARG;
      int64_t nc;
      if (dtype == TSPH_F32) {
        float bf = static_cast<float>(box[k]);
        nc = static_cast<int64_t>(std::floor(bf / static_cast<float>(cutoff)));
        if (nc < 3) nc = 3;
        grid->width[k] = static_cast<double>(bf / static_cast<float>(nc));
      } else {
        nc = static_cast<int64_t>(std::floor(box[k] / cutoff));
        if (nc < 3) nc = 3;
        grid->width[k] = box[k] / static_cast<double>(nc);
      }
      grid->ncell[k] = nc;
      // a wrapped grid has no origin: how far the positions reach, in cutoffs
      const double reach = std::max(std::fabs(static_cast<double>(host[k])), std::fabs(static_cast<double>(host[3 + k]) + 1.0));
      grid->origin[k] = static_cast<int64_t>(std::min(reach, 4.0e18));
    } else {
      grid->origin[k] = n > 0 ? host[k] : 0;
      grid->ncell[k] = n > 0 ? host[3 + k] - host[k] + 1 : 1;
    }
    if (grid->ncell[k] > (int64_t(1) << 31) - 1 || grid->ncell[k] < 1) return TSPH_ERR_GRID;
    cells *= static_cast<double>(grid->ncell[k]);
  }
  if (cells > 9.0e18) return TSPH_ERR_GRID;
  grid->total_cells = grid->ncell[0] * grid->ncell[1] * grid->ncell[2];
  int bits = 0;
  while (bits < 64 && (uint64_t(1) << bits) < static_cast<uint64_t>(grid->total_cells)) ++bits;
  grid->key_bits = bits;
  const int64_t dense_limit = std::max<int64_t>(int64_t(1) << 20, 4 * n);
  grid->dense = grid->total_cells <= dense_limit ? 1 : 0;
  grid->workspace_bytes = static_cast<int64_t>(build_layout(*grid, nullptr, nullptr));
  return TSPH_OK;
}

int64_t tsph_grid_slot_bytes(const tsph_grid* grid, int64_t symmetric) {
  if (!grid || grid->dim < 1 || grid->dim > 3) return 0;
  return grid->n * wanted_slots(*grid, symmetric ? kBoth : kForward) * static_cast<int64_t>(sizeof(uint32_t));
}

int tsph_grid_build(const void* pos, const tsph_grid* grid, void* ws, int64_t ws_bytes,
                    int64_t* order_out, tsph_stream stream) {
  if (!grid) return TSPH_ERR_ARG;
  if (ws_bytes < grid->workspace_bytes) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int64_t n = grid->n;
  if (n == 0) return TSPH_OK;
  BuildWs w;
  build_layout(*grid, &w, ws);
  GridDev g = to_dev(*grid);
  const bool sorted = !grid->dense || order_out != nullptr;
  int rc = TSPH_OK;
  if (sorted) {
    rc = dispatch(grid->dtype, grid->dim, [&](auto t, auto d) {
      using T = decltype(t);
      key_kernel<T, decltype(d)::value><<<grid_for(n, kBlock), kBlock, 0, s>>>(static_cast<const T*>(pos), n, g,
                                                                               w.keys, w.order);
      TSPH_LAUNCH_CHECK();
      return TSPH_OK;
    });
    if (rc) return rc;
    rc = radix_sort_u64_i32(w.keys, w.order, w.keys_tmp, w.order_tmp, n, static_cast<int>(grid->key_bits),
                            w.radix_scratch, s);
    if (rc) return rc;
    if (order_out) {
      order_to_i64<<<grid_for(n, kBlock), kBlock, 0, s>>>(w.order, n, order_out);
      TSPH_LAUNCH_CHECK();
    }
  }
  int32_t* slots = w.order_tmp;
  // the counts and, behind them, what the slots held of earlier positions
  const size_t counts = reinterpret_cast<char*>(w.state + 1) - reinterpret_cast<char*>(w.counts);
  TSPH_CUDA_CHECK(cudaMemsetAsync(w.counts, 0, counts, s));
  return dispatch(grid->dtype, grid->dim, [&](auto t, auto d) -> int {
    using T = decltype(t);
    constexpr int D = decltype(d)::value;
    const T* p = static_cast<const T*>(pos);
    if (grid->dense) {
      cell_count<T, D><<<grid_for(n, kBlock), kBlock, 0, s>>>(p, n, g, w.counts, slots);
      TSPH_LAUNCH_CHECK();
      int rc2 = exclusive_scan_i32_to_i64(w.counts, w.start, grid->total_cells, w.start + grid->total_cells,
                                          w.scan_scratch, s);
      if (rc2) return rc2;
      cell_scatter<T, D, true><<<grid_for(n, kBlock), kBlock, 0, s>>>(p, n, g, w.start, slots, w.order, w.rec,
                                                                          w.cell);
    } else {
      cell_scatter<T, D, false><<<grid_for(n, kBlock), kBlock, 0, s>>>(p, n, g, nullptr, nullptr, w.order, w.rec, w.cell);
    }
    TSPH_LAUNCH_CHECK();
    return TSPH_OK;
  });
}

int tsph_pairs_count(const void* pos, const tsph_grid* grid, int64_t row_limit, void* ws,
                     int64_t ws_bytes, int64_t* pair_count, int64_t* total_count,
                     tsph_stream stream) {
  if (!grid || !pair_count) return TSPH_ERR_ARG;
  if (ws_bytes < grid->workspace_bytes) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int64_t n = grid->n;
  *pair_count = 0;
  if (total_count) *total_count = 0;
  if (n < 2) return TSPH_OK;
  if (row_limit < 0) row_limit = 0;
  if (row_limit > n) row_limit = n;
  BuildWs w;
  build_layout(*grid, &w, ws);
  int rc = count_rows<kForward>(pos, *grid, n, w, row_slots(*grid, kForward, ws_bytes), w.rowptr, s);
  if (rc) return rc;
  int64_t host[2] = {0, 0};
  TSPH_CUDA_CHECK(cudaMemcpyAsync(&host[1], w.rowptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  if (row_limit < n)
    TSPH_CUDA_CHECK(cudaMemcpyAsync(&host[0], w.rowptr + row_limit, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  TSPH_CUDA_CHECK(cudaStreamSynchronize(s));
  if (row_limit == n) host[0] = host[1];
  *pair_count = host[0];
  if (total_count) *total_count = host[1];
  return TSPH_OK;
}

int64_t tsph_pairs_emit_workspace_bytes(int64_t pair_count, int64_t n) {
  (void)n;
  return static_cast<int64_t>(align_up((pair_count + 1) * sizeof(uint32_t)));
}

int tsph_pairs_emit(const void* pos, const tsph_grid* grid, int64_t row_limit, void* ws,
                    int64_t ws_bytes, void* emit_ws, int64_t emit_ws_bytes, int64_t* pairs,
                    int64_t pair_count, tsph_stream stream) {
  if (!grid) return TSPH_ERR_ARG;
  if (ws_bytes < grid->workspace_bytes) return TSPH_ERR_WORKSPACE;
  const int64_t n = grid->n;
  if (pair_count == 0 || n < 2) return TSPH_OK;
  if (emit_ws_bytes < tsph_pairs_emit_workspace_bytes(pair_count, n)) return TSPH_ERR_WORKSPACE;
  if (row_limit < 0) row_limit = 0;
  if (row_limit > n) row_limit = n;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  BuildWs w;
  build_layout(*grid, &w, ws);
  uint32_t* cols = static_cast<uint32_t*>(emit_ws);
  const int slots = row_slots(*grid, kForward, ws_bytes);
  if (reinterpret_cast<uintptr_t>(pairs) % 16 == 0)
    return emit_rows<kForward>(pos, *grid, row_limit, row_limit, w, slots, w.rowptr, cols, pair_count,
                               AsPairs<true>{pairs}, s);
  return emit_rows<kForward>(pos, *grid, row_limit, row_limit, w, slots, w.rowptr, cols, pair_count,
                             AsPairs<false>{pairs}, s);
}

int tsph_rows_count(const void* pos, const tsph_grid* grid, int64_t row_limit, void* ws, int64_t ws_bytes,
                    int64_t* rowptr, int64_t* entry_count, tsph_stream stream) {
  if (!grid || !rowptr || !entry_count) return TSPH_ERR_ARG;
  if (ws_bytes < grid->workspace_bytes) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int64_t n = grid->n;
  *entry_count = 0;
  if (n < 2) {
    TSPH_CUDA_CHECK(cudaMemsetAsync(rowptr, 0, (n + 1) * sizeof(int64_t), s));
    return TSPH_OK;
  }
  BuildWs w;
  build_layout(*grid, &w, ws);
  int rc = count_rows<kBoth>(pos, *grid, std::min(std::max<int64_t>(row_limit, 0), n), w,
                             row_slots(*grid, kBoth, ws_bytes), rowptr, s);
  if (rc) return rc;
  TSPH_CUDA_CHECK(cudaMemcpyAsync(entry_count, rowptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  TSPH_CUDA_CHECK(cudaStreamSynchronize(s));
  return TSPH_OK;
}

int tsph_rows_emit(const void* pos, const tsph_grid* grid, int64_t row_limit, void* ws, int64_t ws_bytes,
                   const int64_t* rowptr, uint32_t* entries, int64_t entry_count, tsph_stream stream) {
  if (!grid) return TSPH_ERR_ARG;
  if (ws_bytes < grid->workspace_bytes) return TSPH_ERR_WORKSPACE;
  const int64_t n = grid->n;
  if (entry_count == 0 || n < 2) return TSPH_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  BuildWs w;
  build_layout(*grid, &w, ws);
  return emit_rows<kBoth>(pos, *grid, std::min(std::max<int64_t>(row_limit, 0), n), n, w,
                          row_slots(*grid, kBoth, ws_bytes), rowptr, entries, entry_count, AsEntries{entries}, s);
}

int64_t tsph_brute_workspace_bytes(int64_t n) {
  return static_cast<int64_t>(align_up((n + 1) * sizeof(int64_t)) + align_up(n * sizeof(int32_t)) +
                              align_up(sizeof(int64_t)) + scan_scratch_bytes(n + 1));
}

int tsph_brute_pairs_count(const void* pos, int64_t n, int64_t dim, int64_t dtype, double cutoff,
                           void* ws, int64_t ws_bytes, int64_t* pair_count, tsph_stream stream) {
  if (ws_bytes < tsph_brute_workspace_bytes(n)) return TSPH_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  *pair_count = 0;
  if (n < 2) return TSPH_OK;
  char* base = static_cast<char*>(ws);
  int64_t* rowptr = reinterpret_cast<int64_t*>(base);
  int32_t* rowcount = reinterpret_cast<int32_t*>(base + align_up((n + 1) * sizeof(int64_t)));
  int64_t* total = reinterpret_cast<int64_t*>(reinterpret_cast<char*>(rowcount) + align_up(n * sizeof(int32_t)));
  char* scan_sc = reinterpret_cast<char*>(total) + align_up(sizeof(int64_t));
  int rc = dispatch(dtype, dim, [&](auto t, auto d) {
    using T = decltype(t);
    brute_kernel<T, decltype(d)::value, 0><<<grid_for(n, 128), 128, 0, s>>>(
        static_cast<const T*>(pos), n, host_cutoff_sq<T>(cutoff), rowcount, nullptr, nullptr);
    TSPH_LAUNCH_CHECK();
    return TSPH_OK;
  });
  if (rc) return rc;
  rc = exclusive_scan_i32_to_i64(rowcount, rowptr, n, total, scan_sc, s);
  if (rc) return rc;
  TSPH_CUDA_CHECK(cudaMemcpyAsync(pair_count, total, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  TSPH_CUDA_CHECK(cudaStreamSynchronize(s));
  return TSPH_OK;
}

int tsph_brute_pairs_emit(const void* pos, int64_t n, int64_t dim, int64_t dtype, double cutoff,
                          void* ws, int64_t ws_bytes, int64_t* pairs, int64_t pair_count,
                          tsph_stream stream) {
  if (ws_bytes < tsph_brute_workspace_bytes(n)) return TSPH_ERR_WORKSPACE;
  if (pair_count == 0 || n < 2) return TSPH_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int64_t* rowptr = static_cast<int64_t*>(ws);
  return dispatch(dtype, dim, [&](auto t, auto d) {
    using T = decltype(t);
    brute_kernel<T, decltype(d)::value, 1><<<grid_for(n, 128), 128, 0, s>>>(
        static_cast<const T*>(pos), n, host_cutoff_sq<T>(cutoff), nullptr, rowptr, pairs);
    TSPH_LAUNCH_CHECK();
    return TSPH_OK;
  });
}

int tsph_max_displacement(const void* pos, const void* anchor, int64_t n, int64_t dim,
                          int64_t dtype, const double* box, double* out, tsph_stream stream) {
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  TSPH_CUDA_CHECK(cudaMemsetAsync(out, 0, sizeof(double), s));
  if (n == 0) return TSPH_OK;
  double b[3] = {1, 1, 1};
  if (box)
    for (int k = 0; k < dim; ++k) b[k] = box[k];
  return dispatch(dtype, dim, [&](auto t, auto d) {
    using T = decltype(t);
    displacement_kernel<T, decltype(d)::value><<<grid_for(n, kBlock, 148 * 8), kBlock, 0, s>>>(
        static_cast<const T*>(pos), static_cast<const T*>(anchor), n, box != nullptr, b[0], b[1], b[2],
        reinterpret_cast<unsigned long long*>(out));
    TSPH_LAUNCH_CHECK();
    return TSPH_OK;
  });
}

}  // extern "C"
