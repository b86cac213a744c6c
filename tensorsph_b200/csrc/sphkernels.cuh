// Smoothing kernels evaluated per pair inside the gather loops.
//
// Cubic spline (Monaghan 1992), support 2h, q = r / h:
//   f(q)  = 1 - 1.5 q^2 + 0.75 q^3      (q < 1)
//         = 0.25 (2 - q)^3              (1 <= q < 2)
//   f'(q) = -3 q + 2.25 q^2 | -0.75 (2 - q)^2
//   f''(q)= -3 + 4.5 q      | 1.5 (2 - q)
// W = sigma f(q), grad_i W = delta * sigma f'(q) / (h max(r, eps)),
// 3-D Laplacian = sigma (f'' + 2 f'/q) / h^2 with the q -> 0 limit -6 for
// 2 f'/q (droplet_impact.py:276-371, threed/kernel3.py:48-181).
// Wendland C2: f = (1 - q/2)^4 (2 q + 1), f' = -5 q (1 - q/2)^3
// (droplet_impact.py:320-346).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace tsph {

template <class T>
struct Cubic {
  T inv_h, h, sigma, eps;
  T inv_lo;    // 1 / h = inv_h + inv_lo (FP32; 0 in FP64)
  T sigma_h;   // sigma / h
  T sigma_hh;  // sigma / h^2
  T sigma_lo;  // sigma to twice the precision: sigma + sigma_lo (FP32; 0 in FP64)
  // Both branches and a select: the neighbours of a warp lie on both sides.
  __device__ __forceinline__ T shape(T q) const {
    const T t = T(2) - q;
    const T near = T(1) - T(1.5) * q * q + T(0.75) * q * q * q, far = T(0.25) * t * t * t;
    return q < T(1) ? near : (q < T(2) ? far : T(0));
  }
  __device__ __forceinline__ T dshape(T q) const {
    const T t = T(2) - q;
    const T near = T(-3) * q + T(2.25) * q * q, far = T(-0.75) * t * t;
    return q < T(1) ? near : (q < T(2) ? far : T(0));
  }
  // W(r)
  __device__ __forceinline__ T w(T r) const {
    T s = shape(r / h);
    return sigma * (s > T(0) ? s : T(0));
  }
  // W(r) and the gradient scale g such that grad_i W = delta * g.
  __device__ __forceinline__ void wg(T r, T& W, T& g) const {
    T q = r / h;
    T s = shape(q);
    W = sigma * (s > T(0) ? s : T(0));
    g = sigma * dshape(q) / (h * (r > eps ? r : eps));
  }
  // W and g from r^2, without the divisions r / h and 1 / (h r).  In FP32 1 / h
  // is a sum of two floats: the rounding of a single one (or of h) stretches
  // every q of a call alike, and that common error, not the terms' own, is most
  // of a density's (measured: 4e-8 to 1.8e-7 of rho0 as 1 / h happens to round).
  // 1 / r is a reciprocal square root (2 ulp in FP32, 1 in FP64, where it gives
  // r as well).
  __device__ __forceinline__ T scaled(T r) const {
    return sizeof(T) == 8 ? r * inv_h : fma(r, inv_h, r * inv_lo);
  }
  __device__ __forceinline__ T shape2(T r2) const { return shape(sizeof(T) == 8 ? radial(r2).q : scaled(sqrt(r2))); }
  __device__ __forceinline__ T w2(T r2) const {
    const T s = shape2(r2);
    return sigma * (s > T(0) ? s : T(0));
  }
  // sigma times a sum of shapes, rounded once
  __device__ __forceinline__ T times_sigma(const CSum<double>& s) const { return sigma * s.s; }
  __device__ __forceinline__ T times_sigma(const CSum<float>& s) const {
    return fma(s.s, sigma, fma(s.s, sigma_lo, s.c * sigma));
  }
  // q = r / h and 1 / max(r, eps).  For r < eps in FP64 q is r^2 / (eps h), as
  // good as r / h there: f is 1 to the last bit and f' too small to matter.
  struct Radial {
    T q, ir;
  };
  __device__ __forceinline__ Radial radial(T r2) const {
    const T ir = r2 > eps * eps ? rsqrt(r2) : T(1) / eps;
    return Radial{scaled(sizeof(T) == 8 ? r2 * ir : sqrt(r2)), ir};
  }
  // The gradient scale g (grad_i W = delta * g) and, with it, W.
  __device__ __forceinline__ T g2(const Radial& R) const { return sigma_h * dshape(R.q) * R.ir; }
  __device__ __forceinline__ void wg2(T r2, T& W, T& g) const {
    const Radial R = radial(r2);
    const T s = shape(R.q);
    W = sigma * (s > T(0) ? s : T(0));
    g = g2(R);
  }
  // 3-D Laplacian of W (threed/kernel3.py:108-124): sigma / h^2 (f'' + 2 f' / q) with the
  // quotient written out (f' / q = -3 + 2.25 q below q = 1, its limit at 0 included).
  __device__ __forceinline__ T lap2(const Radial& R) const {
    const T t = T(2) - R.q;
    const T near = T(-9) + T(9) * R.q, far = t * (T(1.5) - T(1.5) * t * (h * R.ir));
    return sigma_hh * (R.q < T(1) ? near : (R.q < T(2) ? far : T(0)));
  }
};

template <class T>
__host__ inline Cubic<T> make_cubic(double h, double sigma) {
  Cubic<T> k;
  k.h = static_cast<T>(h);
  k.inv_h = static_cast<T>(1.0 / h);
  k.inv_lo = static_cast<T>(1.0 / h - static_cast<double>(k.inv_h));
  k.sigma = static_cast<T>(sigma);
  k.sigma_h = static_cast<T>(sigma / h);
  k.sigma_hh = static_cast<T>(sigma / (h * h));
  k.sigma_lo = static_cast<T>(sigma - static_cast<double>(k.sigma));
  k.eps = static_cast<T>(1e-12);
  return k;
}

template <class T>
struct Wendland {
  T h, sigma, eps;
  __device__ __forceinline__ T w(T r) const {
    T q = r / h;
    T t = T(1) - T(0.5) * q;
    t = t > T(0) ? t : T(0);
    T t2 = t * t;
    return sigma * t2 * t2 * (T(2) * q + T(1));
  }
  __device__ __forceinline__ void wg(T r, T& W, T& g) const {
    T q = r / h;
    T t = T(1) - T(0.5) * q;
    t = t > T(0) ? t : T(0);
    T t2 = t * t;
    W = sigma * t2 * t2 * (T(2) * q + T(1));
    g = sigma * (T(-5) * q * t2 * t) / (h * (r > eps ? r : eps));
  }
};

}  // namespace tsph
