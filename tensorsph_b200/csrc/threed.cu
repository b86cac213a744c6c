// Fused gather kernels of tensorsph.threed.accelerations (operators3.py:212-256).
//
//   T1 density     rho_a = sum_b m_b W_ab + m_a W(0)                     all rows
//   T2 gradient    <grad rho> for the Antuono psi form (fluid rows, fluid pairs)
//   T3 diffusion   rho_a = max(rho_a + dt rate_a, 0.1 rho0), Tait p        all rows
//   T4 walls       Adami p_w = sum_f (p_f + rho_f g.(x_w - x_f)) W / sum W  wall rows
//   T5 moments     K_a = 1/3 sum_b V r^2 lap W (+ I4 for order 4)           all rows
//   T6 force       pressure + renormalised Brookshaw Laplacian + g          all rows
//   T7 order 4     a_a -= nu sum_b w beta (L_b - L_a)                       all rows
// Separations use the minimum image when a periodic box is given; the Adami
// weights use the plain distance, as the reference does (operators3.py:195-197).
//
// Two to eight lanes share a row (gather.cuh).  What bounds the passes: FP64
// (or FP32) instruction issue.  m / rho and p / rho^2 are formed once per
// particle, the image of a separation needs no division for a neighbour, and
// the kernel terms come from one reciprocal square root.
#include <cmath>

#include "common.cuh"
#include "fpmath.cuh"
#include "gather.cuh"
#include "sphkernels.cuh"
#include "symeig.cuh"

namespace tsph {
namespace {

constexpr uint32_t kSecond = 0x80000000u;

template <class T>
struct TP {
  int64_t n, nf;
  int periodic, has_g, renorm, order, diffusion, form, adami;
  T box[3], half[3], g[3];
  T rho0, bulk, gamma, inv_gamma, nu, dt, dscale, rho_floor, eigen_floor;
  Cubic<T> k;
};

template <class T>
__device__ __forceinline__ void sep(const Q4<T>& a, const Q4<T>& b, const TP<T>& p, T d[3]) {
  d[0] = a.x - b.x;
  d[1] = a.y - b.y;
  d[2] = a.z - b.z;
  // most neighbours need no image on any axis
  if (p.periodic && !(fabs(d[0]) <= p.half[0] && fabs(d[1]) <= p.half[1] && fabs(d[2]) <= p.half[2])) {
#pragma unroll
    for (int k = 0; k < 3; ++k) d[k] = fp<T>::min_image(d[k], p.box[k]);
  }
}

template <class T>
__device__ __forceinline__ T tait3(T rho, const TP<T>& p) {
  T v = p.bulk * (pow(rho / p.rho0, p.gamma) - T(1));
  return v > T(0) ? v : T(0);
}

template <class T>
__device__ __forceinline__ T dot3(const T a[3], const T b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

template <class T>
__global__ void t_pack(const T* __restrict__ pos, const T* __restrict__ vel, const T* __restrict__ mass,
                       int64_t n, Q4<T>* __restrict__ pm, Q4<T>* __restrict__ vv) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < n;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    pm[a] = Q4<T>{pos[3 * a], pos[3 * a + 1], pos[3 * a + 2], mass[a]};
    vv[a] = Q4<T>{vel[3 * a], vel[3 * a + 1], vel[3 * a + 2], T(0)};
  }
}

// rv: (rho before diffusion, m / rho); st: (rho, p) when there is no diffusion.
template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_density(TP<T> p, const Q4<T>* __restrict__ pm,
                                                          const int64_t* __restrict__ rowptr,
                                                          const uint32_t* __restrict__ ent, Q2<T>* __restrict__ rv,
                                                          Q2<T>* __restrict__ st) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= p.n) return;
  const Q4<T> pa = pm[a];
  CSum<T> s;
  me.walk_ahead(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const Q4<T> pb = pm[e & kIndexMask];
    T d[3];
    sep(pa, pb, p, d);
    s.add(pb.w * p.k.shape2(dot3(d, d)));
  });
  if (me.lane == 0) s.add(pa.w);  // W(0) = sigma
  const T r = p.k.times_sigma(me.total(s));
  if (me.lane) return;
  if (p.diffusion)
    rv[a] = Q2<T>{r, pa.w / r};
  else
    st[a] = Q2<T>{r, tait3(r, p)};
}

template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_gradient(TP<T> p, const Q4<T>* __restrict__ pm,
                                                           const int64_t* __restrict__ rowptr,
                                                           const uint32_t* __restrict__ ent,
                                                           const Q2<T>* __restrict__ rv, Q4<T>* __restrict__ grad) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= p.nf) return;
  const Q4<T> pa = pm[a];
  const T ra = rv[a].x;
  CSum<T> G[3], M[6];
  me.walk_ahead(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const uint32_t b = e & kIndexMask;
    if (b >= p.nf) return;
    const Q4<T> pb = pm[b];
    const Q2<T> sb = rv[b];
    T d[3];
    sep(pa, pb, p, d);
    const T gs = p.k.g2(p.k.radial(dot3(d, d)));
    const T vb = sb.y, diff = sb.x - ra;
    const T g[3] = {d[0] * gs, d[1] * gs, d[2] * gs};
#pragma unroll
    for (int r = 0; r < 3; ++r) G[r].add(vb * diff * g[r]);
    M[0].add(vb * -(d[0] * g[0]));
    M[1].add(vb * -(d[1] * g[0]));
    M[2].add(vb * -(d[1] * g[1]));
    M[3].add(vb * -(d[2] * g[0]));
    M[4].add(vb * -(d[2] * g[1]));
    M[5].add(vb * -(d[2] * g[2]));
  });
  double m[3][3], rhs[3], out[3];
  m[0][0] = me.sum(M[0]);
  m[1][0] = m[0][1] = me.sum(M[1]);
  m[1][1] = me.sum(M[2]);
  m[2][0] = m[0][2] = me.sum(M[3]);
  m[2][1] = m[1][2] = me.sum(M[4]);
  m[2][2] = me.sum(M[5]);
  for (int r = 0; r < 3; ++r) rhs[r] = me.sum(G[r]);
  if (me.lane) return;
  floored_solve<3>(m, rhs, static_cast<double>(p.eigen_floor), out);
  grad[a] = Q4<T>{static_cast<T>(out[0]), static_cast<T>(out[1]), static_cast<T>(out[2]), T(0)};
}

template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_diffusion(TP<T> p, const Q4<T>* __restrict__ pm,
                                                            const int64_t* __restrict__ rowptr,
                                                            const uint32_t* __restrict__ ent,
                                                            const Q2<T>* __restrict__ rv,
                                                            const Q4<T>* __restrict__ grad, Q2<T>* __restrict__ st) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= p.n) return;
  const T ra = rv[a].x;
  CSum<T> rate;
  if (a < p.nf) {
    const Q4<T> pa = pm[a];
    const Q4<T> ga = p.form == 1 ? grad[a] : Q4<T>{T(0), T(0), T(0), T(0)};
    me.walk_ahead(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
      const uint32_t b = e & kIndexMask;
      if (b >= p.nf) return;
      const Q4<T> pb = pm[b];
      const Q2<T> sb = rv[b];
      T d[3];
      sep(pa, pb, p, d);
      const T d2 = dot3(d, d);
      const T gs = p.k.g2(p.k.radial(d2));
      const T radial = -(d[0] * (d[0] * gs) + d[1] * (d[1] * gs) + d[2] * (d[2] * gs));
      T contrast = ra - sb.x;
      if (p.form == 1) {
        const Q4<T> gb = grad[b];
        const T proj = (ga.x + gb.x) * d[0] + (ga.y + gb.y) * d[1] + (ga.z + gb.z) * d[2];
        contrast = contrast - T(0.5) * proj;
      }
      const T coupling = contrast * radial / (d2 + T(1e-12));
      rate.add((-p.dscale * sb.y) * coupling);
    });
  }
  const T rate_v = me.sum(rate);
  if (me.lane) return;
  T r = ra + p.dt * rate_v;
  r = r > p.rho_floor ? r : p.rho_floor;
  st[a] = Q2<T>{r, tait3(r, p)};
}

// ru: the walls' density of the Tait inverse, which the force uses instead of
// their summed one.
template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_walls(TP<T> p, const Q4<T>* __restrict__ pm,
                                                        const int64_t* __restrict__ rowptr,
                                                        const uint32_t* __restrict__ ent, Q2<T>* st,
                                                        T* __restrict__ ru) {
  const RowLanes<L> me;
  const int64_t a = p.nf + me.row;
  if (a >= p.n) return;
  const Q4<T> pa = pm[a];
  CSum<T> num, den;
  me.walk_ahead(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const uint32_t f = e & kIndexMask;
    if (f >= p.nf) return;
    const Q4<T> pb = pm[f];
    const Q2<T> sf = st[f];
    const T d[3] = {pa.x - pb.x, pa.y - pb.y, pa.z - pb.z};  // x_w - x_f, no image
    const T W = p.k.w2(dot3(d, d));
    T donor = sf.y;
    if (p.has_g) donor = donor + sf.x * dot3(d, p.g);
    num.add(donor * W);
    den.add(W);
  });
  const T dd = me.sum(den), nn = me.sum(num);
  if (me.lane) return;
  T pw = dd > T(0) ? nn / (dd > T(1e-30) ? dd : T(1e-30)) : T(0);
  pw = pw > T(0) ? pw : T(0);
  st[a].y = pw;
  ru[a - p.nf] = p.rho0 * pow(T(1) + pw / p.bulk, p.inv_gamma);
}

// rho and p out; st becomes (rho_used, p / rho_used^2), rho_used the density
// (the walls' own under the Adami model).
template <class T>
__global__ void t_state(TP<T> p, const T* __restrict__ ru, Q2<T>* __restrict__ st, T* __restrict__ rho,
                        T* __restrict__ pressure) {
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < p.n;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const Q2<T> s = st[a];
    rho[a] = s.x;
    pressure[a] = s.y;
    const T r = p.adami && a >= p.nf ? ru[a - p.nf] : s.x;
    st[a] = Q2<T>{r, s.y / (r * r)};
  }
}

// K goes to the fourth place of the velocity record, where the force reads it.
template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_moments(TP<T> p, const Q4<T>* __restrict__ pm,
                                                          const int64_t* __restrict__ rowptr,
                                                          const uint32_t* __restrict__ ent,
                                                          const Q2<T>* __restrict__ st, Q4<T>* __restrict__ vv,
                                                          T* __restrict__ I4) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= p.n) return;
  const Q4<T> pa = pm[a];
  const T ra = st[a].x;
  CSum<T> k2, k4;
  me.walk_ahead(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const uint32_t b = e & kIndexMask;
    const Q4<T> pb = pm[b];
    T d[3];
    sep(pa, pb, p, d);
    const T r2 = dot3(d, d);
    const T lap = p.k.lap2(p.k.radial(r2));
    const T term = r2 * lap * pb.w / (T(0.5) * (ra + st[b].x));
    k2.add(term);
    if (p.order == 4) k4.add(r2 * term);
  });
  const T s2 = me.sum(k2), s4 = p.order == 4 ? me.sum(k4) : T(0);
  if (me.lane) return;
  vv[a].w = s2 / T(3);
  if (p.order == 4) I4[a] = s4;
}

// Pair weight of the Brookshaw operator: the reference multiplies by the mass
// of the pair's *second* element (operators3.py:137), kept per entry flag.
template <class T>
__device__ __forceinline__ T brook_weight(const TP<T>& p, uint32_t e, const Q4<T>& pa, const Q4<T>& pb,
                                          T lap, T rbar, T Ka, T Kb) {
  const T m_second = (e & kSecond) ? pa.w : pb.w;
  if (!p.renorm) return m_second * lap / rbar;
  const T kb = T(0.5) * (Ka + Kb);
  return T(2) * (m_second * lap) / (rbar * (kb > T(1e-12) ? kb : T(1e-12)));
}

template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_force(TP<T> p, const Q4<T>* __restrict__ pm,
                                                        const Q4<T>* __restrict__ vv,
                                                        const int64_t* __restrict__ rowptr,
                                                        const uint32_t* __restrict__ ent,
                                                        const Q2<T>* __restrict__ st, T* __restrict__ acc,
                                                        Q4<T>* __restrict__ lap1) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= p.n) return;
  const Q4<T> pa = pm[a], va = vv[a];
  const Q2<T> sa = st[a];
  CSum<T> ax, ay, az, lx, ly, lz;
  const bool viscous = p.nu != T(0);
  me.walk(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const uint32_t b = e & kIndexMask;
    const Q4<T> pb = pm[b];
    const Q2<T> sb = st[b];
    T d[3];
    sep(pa, pb, p, d);
    const auto R = p.k.radial(dot3(d, d));
    const T gs = p.k.g2(R);
    const T c = -pb.w * (sa.y + sb.y);
    ax.add(d[0] * gs * c);
    ay.add(d[1] * gs * c);
    az.add(d[2] * gs * c);
    if (viscous) {
      const Q4<T> vb = vv[b];
      const T w = brook_weight(p, e, pa, pb, p.k.lap2(R), T(0.5) * (sa.x + sb.x), va.w, vb.w);
      lx.add((vb.x - va.x) * w);
      ly.add((vb.y - va.y) * w);
      lz.add((vb.z - va.z) * w);
    }
  });
  T out[3] = {me.sum(ax), me.sum(ay), me.sum(az)};
  T lap[3] = {T(0), T(0), T(0)};
  if (viscous) {
    lap[0] = me.sum(lx);
    lap[1] = me.sum(ly);
    lap[2] = me.sum(lz);
  }
  if (me.lane) return;
  if (viscous) {
    if (p.order == 4) {
      lap1[a] = Q4<T>{lap[0], lap[1], lap[2], T(0)};
    } else {
      for (int k = 0; k < 3; ++k) out[k] = out[k] + lap[k] * p.nu;
    }
  }
  if (p.order != 4 || !viscous) {
    if (p.has_g && a < p.nf)
      for (int k = 0; k < 3; ++k) out[k] = out[k] + p.g[k];
  }
  for (int k = 0; k < 3; ++k) acc[3 * a + k] = out[k];
}

template <class T, int L>
__global__ void __launch_bounds__(kGatherBlock) t_order4(TP<T> p, const Q4<T>* __restrict__ pm,
                                                         const Q4<T>* __restrict__ vv,
                                                         const int64_t* __restrict__ rowptr,
                                                         const uint32_t* __restrict__ ent,
                                                         const Q2<T>* __restrict__ st, const T* __restrict__ I4,
                                                         const Q4<T>* __restrict__ lap1, T* __restrict__ acc) {
  const RowLanes<L> me;
  const int64_t a = me.row;
  if (a >= p.n) return;
  const Q4<T> pa = pm[a], la = lap1[a];
  const T ra = st[a].x, Ka = vv[a].w, ia = I4[a];
  CSum<T> lx, ly, lz;
  me.walk(ent, rowptr[a], rowptr[a + 1], [&](uint32_t e) {
    const uint32_t b = e & kIndexMask;
    const Q4<T> pb = pm[b], lb = lap1[b];
    T d[3];
    sep(pa, pb, p, d);
    const T lap = p.k.lap2(p.k.radial(dot3(d, d)));
    const T w = brook_weight(p, e, pa, pb, lap, T(0.5) * (ra + st[b].x), Ka, vv[b].w);
    const T wb = w * (T(0.5) * (ia + I4[b]) / T(120));
    lx.add((lb.x - la.x) * wb);
    ly.add((lb.y - la.y) * wb);
    lz.add((lb.z - la.z) * wb);
  });
  const T corr[3] = {me.sum(lx), me.sum(ly), me.sum(lz)};
  if (me.lane) return;
  const T l0[3] = {la.x, la.y, la.z};
  for (int k = 0; k < 3; ++k) {
    T v = acc[3 * a + k] + (l0[k] - corr[k]) * p.nu;
    if (p.has_g && a < p.nf) v = v + p.g[k];
    acc[3 * a + k] = v;
  }
}

struct TLayout {
  size_t pm, vv, rv, st, ru, I4, grad, lap1, total;
};

TLayout t_layout(const tsph_threed_params& prm) {
  const size_t ts = prm.dtype == TSPH_F64 ? 8 : 4;
  const int64_t n = prm.n;
  TLayout L{};
  size_t off = 0;
  L.pm = off; off += align_up(n * 4 * ts);
  L.vv = off; off += align_up(n * 4 * ts);
  L.rv = off; off += align_up(n * 2 * ts);
  L.st = off; off += align_up(n * 2 * ts);
  L.ru = off; off += align_up(n * ts);
  L.I4 = off; off += align_up(n * ts);
  L.grad = L.lap1 = off; off += align_up(n * 4 * ts);  // lap1 after the diffusion is done with grad
  L.total = off + 256;
  return L;
}

template <class T, int LN>
int run_rows(const tsph_threed_params& prm, const tsph_threed_io& io, char* ws, cudaStream_t s) {
  TLayout L = t_layout(prm);
  Q4<T>* pm = reinterpret_cast<Q4<T>*>(ws + L.pm);
  Q4<T>* vv = reinterpret_cast<Q4<T>*>(ws + L.vv);
  Q2<T>* rv = reinterpret_cast<Q2<T>*>(ws + L.rv);
  Q2<T>* st = reinterpret_cast<Q2<T>*>(ws + L.st);
  T* ru = reinterpret_cast<T*>(ws + L.ru);
  T* I4 = reinterpret_cast<T*>(ws + L.I4);
  Q4<T>* grad = reinterpret_cast<Q4<T>*>(ws + L.grad);
  Q4<T>* lap1 = reinterpret_cast<Q4<T>*>(ws + L.lap1);
  const int64_t n = prm.n, nf = prm.n_fluid;

  TP<T> p{};
  p.n = n;
  p.nf = nf;
  p.periodic = static_cast<int>(prm.periodic);
  p.has_g = static_cast<int>(prm.has_gravity);
  p.renorm = static_cast<int>(prm.renormalise);
  p.order = static_cast<int>(prm.viscous_order);
  p.diffusion = prm.diffusion > 0.0;
  p.form = static_cast<int>(prm.diffusion_form);
  p.adami = nf < n && prm.wall_model == 0;
  for (int k = 0; k < 3; ++k) {
    p.box[k] = static_cast<T>(prm.box[k]);
    p.half[k] = T(0.5) * p.box[k];
    p.g[k] = static_cast<T>(prm.gravity[k]);
  }
  p.rho0 = static_cast<T>(prm.rho0);
  p.bulk = static_cast<T>(prm.rho0 * prm.sound_speed * prm.sound_speed / prm.gamma);
  p.gamma = static_cast<T>(prm.gamma);
  p.inv_gamma = static_cast<T>(1.0 / prm.gamma);
  p.nu = static_cast<T>(prm.viscosity);
  p.dt = static_cast<T>(prm.dt);
  p.dscale = static_cast<T>(2.0 * prm.diffusion * prm.sound_speed * prm.h);
  p.rho_floor = static_cast<T>(0.1 * prm.rho0);
  const double sigma = 1.0 / (M_PI * prm.h * prm.h * prm.h);
  p.eigen_floor = static_cast<T>(prm.eigen_floor);
  p.k = make_cubic<T>(prm.h, sigma);

  constexpr int B = kGatherBlock;
  const unsigned g = row_grid(n, LN);
  t_pack<T><<<grid_for(n, 256), 256, 0, s>>>(static_cast<const T*>(io.pos), static_cast<const T*>(io.vel),
                                              static_cast<const T*>(io.mass), n, pm, vv);
  TSPH_LAUNCH_CHECK();
  t_density<T, LN><<<g, B, 0, s>>>(p, pm, io.rowptr, io.entries, rv, st);
  TSPH_LAUNCH_CHECK();
  if (p.diffusion) {
    if (p.form == 1) {
      t_gradient<T, LN><<<row_grid(nf, LN), B, 0, s>>>(p, pm, io.rowptr, io.entries, rv, grad);
      TSPH_LAUNCH_CHECK();
    }
    t_diffusion<T, LN><<<g, B, 0, s>>>(p, pm, io.rowptr, io.entries, rv, grad, st);
    TSPH_LAUNCH_CHECK();
  }
  if (p.adami) {
    t_walls<T, LN><<<row_grid(n - nf, LN), B, 0, s>>>(p, pm, io.rowptr, io.entries, st, ru);
    TSPH_LAUNCH_CHECK();
  }
  t_state<T><<<grid_for(n, 256), 256, 0, s>>>(p, ru, st, static_cast<T*>(io.rho), static_cast<T*>(io.pressure));
  TSPH_LAUNCH_CHECK();
  if (p.nu != T(0)) {
    t_moments<T, LN><<<g, B, 0, s>>>(p, pm, io.rowptr, io.entries, st, vv, I4);
    TSPH_LAUNCH_CHECK();
  }
  t_force<T, LN><<<g, B, 0, s>>>(p, pm, vv, io.rowptr, io.entries, st, static_cast<T*>(io.acc), lap1);
  TSPH_LAUNCH_CHECK();
  if (p.nu != T(0) && p.order == 4) {
    t_order4<T, LN><<<g, B, 0, s>>>(p, pm, vv, io.rowptr, io.entries, st, I4, lap1, static_cast<T*>(io.acc));
    TSPH_LAUNCH_CHECK();
  }
  return TSPH_OK;
}

template <class T>
int run_threed(const tsph_threed_params& prm, const tsph_threed_io& io, char* ws, cudaStream_t s) {
  return with_lanes<3>(prm.n, [&](auto lanes) { return run_rows<T, decltype(lanes)::value>(prm, io, ws, s); });
}

}  // namespace
}  // namespace tsph

using namespace tsph;

extern "C" {

int64_t tsph_threed_workspace_bytes(const tsph_threed_params* prm) {
  if (!prm) return -1;
  return static_cast<int64_t>(t_layout(*prm).total);
}

int tsph_threed_accelerations(const tsph_threed_params* prm, const tsph_threed_io* io, void* ws,
                              int64_t ws_bytes, tsph_stream stream) {
  if (!prm || !io) return TSPH_ERR_ARG;
  if (prm->n < 0 || prm->n_fluid < 0 || prm->n_fluid > prm->n || prm->n >= (int64_t(1) << 31))
    return TSPH_ERR_ARG;
  if (prm->viscous_order != 2 && prm->viscous_order != 4) return TSPH_ERR_ARG;
  if (prm->wall_model != 0 && prm->wall_model != 1) return TSPH_ERR_ARG;
  if (ws_bytes < tsph_threed_workspace_bytes(prm)) return TSPH_ERR_WORKSPACE;
  if (prm->n == 0) return TSPH_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (prm->dtype == TSPH_F32) return run_threed<float>(*prm, *io, static_cast<char*>(ws), s);
  if (prm->dtype == TSPH_F64) return run_threed<double>(*prm, *io, static_cast<char*>(ws), s);
  return TSPH_ERR_ARG;
}

}  // extern "C"
