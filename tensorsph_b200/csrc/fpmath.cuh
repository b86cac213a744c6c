// IEEE round-to-nearest arithmetic with no contraction, per dtype.
//
// The reference evaluates every elementwise op as a separately rounded
// PyTorch kernel; where integer results (cell keys, pair membership) depend on
// the last bit, the CUDA path uses the same rounded operations.
#pragma once

#include <cuda_runtime.h>

namespace tsph {

template <class T>
struct fp;

// delta - box * round_half_even(delta / box)  (threed/neighbors3.py:45-53),
// without its division where the rounded quotient is plain: |d| <= box / 2
// rounds to 0 (d / box is at most 1/2 after rounding, and 1/2 rounds to even),
// and 0.6 box <= |d| <= 1.4 box to +-1 (the quotient is within 0.59 .. 1.41).
// A neighbour pair across a box of three cutoffs or more is always one of the
// two; the division is 3 of the ~10 FP64 divisions of a periodic pair term.
template <class F, class T>
__device__ __forceinline__ T image(T d, T box) {
  const T a = fabs(d);
  if (a <= T(0.5) * box) return d;
  if (a >= T(0.6) * box && a <= T(1.4) * box) return F::sub(d, copysign(box, d));
  return F::sub(d, F::mul(box, F::rint(F::div(d, box))));
}

template <>
struct fp<float> {
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
  static __device__ __forceinline__ float sqrt(float a) { return __fsqrt_rn(a); }
  static __device__ __forceinline__ float rint(float a) { return rintf(a); }
  static __device__ __forceinline__ float min_image(float d, float box) { return image<fp<float>>(d, box); }
};

template <>
struct fp<double> {
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
  static __device__ __forceinline__ double sqrt(double a) { return __dsqrt_rn(a); }
  static __device__ __forceinline__ double rint(double a) { return ::rint(a); }
  static __device__ __forceinline__ double min_image(double d, double box) { return image<fp<double>>(d, box); }
};

}  // namespace tsph
