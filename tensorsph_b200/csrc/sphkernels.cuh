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

namespace tsph {

template <class T>
struct Cubic {
  T inv_h, h, sigma, eps;
  T inv_lo;    // 1 / h = inv_h + inv_lo (FP32; 0 in FP64)
  T sigma_h;   // sigma / h
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
  // r as well).  Below eps, where g is a division by eps, w() and wg().
  __device__ __forceinline__ T scaled(T r) const {
    return sizeof(T) == 8 ? r * inv_h : fma(r, inv_h, r * inv_lo);
  }
  __device__ __forceinline__ T shape2(T r2) const { return shape(scaled(sqrt(r2))); }
  __device__ __forceinline__ T w2(T r2) const {
    const T s = shape2(r2);
    return sigma * (s > T(0) ? s : T(0));
  }
  // sigma times a sum of shapes
  __device__ __forceinline__ T times_sigma(T s) const { return sizeof(T) == 8 ? sigma * s : fma(s, sigma, s * sigma_lo); }
  __device__ __forceinline__ void wg2(T r2, T& W, T& g) const {
    if (r2 > eps * eps) {
      const T ir = rsqrt(r2), q = scaled(sizeof(T) == 8 ? r2 * ir : sqrt(r2)), s = shape(q);
      W = sigma * (s > T(0) ? s : T(0));
      g = sigma_h * dshape(q) * ir;
    } else {
      wg(sqrt(r2), W, g);
    }
  }
  // 3-D Laplacian of W (threed/kernel3.py:108-124).
  __device__ __forceinline__ T lap3(T r) const {
    T q = r / h;
    if (!(q < T(2))) return T(0);
    T second = q < T(1) ? T(-3) + T(4.5) * q : T(1.5) * (T(2) - q);
    T twice = q > T(1e-10) ? T(2) * dshape(q) / (q > eps ? q : eps) : T(-6);
    return sigma * (second + twice) / (h * h);
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
