// The reference's cubic interpolant of pixels (CubicInterpolate,
// src/interpol.cpp:42-53) in fewer instructions and the same bits.  Files that
// include this header are compiled with -fmad=false: the fused multiply-adds
// here are written out, and their products are exact.
#pragma once

#include <cuda_runtime.h>

namespace ptk {

// exact uint16 -> double without the conversion pipe: the bits of 2^52 + v, minus 2^52
__device__ __forceinline__ double u16d(unsigned v) { return __hiloint2double(0x43300000, (int)v) - 0x1p52; }

// floor(x) and x - floor(x), both exact, for 0 <= x < 2^31: the nearest
// integer in the low mantissa bits of x + 1.5 * 2^52, one less where it lies
// above x.
__device__ __forceinline__ double split(double x, int* ix) {
  const double t = x + 0x1.8p52;
  const double f = x - (t - 0x1.8p52);  // in [-0.5, 0.5]
  const int below = __double2hiint(f) < 0 ? 1 : 0;  // (x an integer: f = +0)
  *ix = __double2loint(t) - below;
  return f + __hiloint2double(below ? 0x3ff00000 : 0, 0);
}

// Twice cubic1 of four pixels at x (x2 = x * x): its coefficients are multiples
// of 1/2 below 2^20, which cubic1's operations reach without rounding, so they
// are formed as integers, doubled; twice every later operation's value is that
// operation on doubled values.  The conversions run on their own pipe, at an
// eighth of the FP64 rate but in one instruction each: with 18 a point, their
// pipe is as busy as the FP64 one.  (Through the bits of 2^52 + v, which takes
// three instructions, an evaluation issued 397 instructions per warp and point
// in all, 122 of them FP64, instead of 357 and 105: 400 grains 7.77 -> 7.63 ms,
// 2000 27.2 -> 26.5 ms.)
__device__ __forceinline__ double cubic_px_twice(int p0, int p1, int p2, int p3, double x, double x2) {
  const int d = p1 - p2, t = p3 - p0;
  const double a = (double)(3 * d + t);
  const double b = (double)(p0 - p1 - t - 4 * d);
  const double c = (double)(p2 - p0);
  return __fma_rn(2.0, (double)p1, a * x2 * x + b * x2 + c * x);
}

// cubic_px_twice, and twice the derivative with respect to x:
// 3 a x x + 2 b x + c in that order.
__device__ __forceinline__ double cubic_px_twice(int p0, int p1, int p2, int p3, double x, double x2, double* dx) {
  const int d = p1 - p2, t = p3 - p0;
  const double a = (double)(3 * d + t);
  const double b = (double)(p0 - p1 - t - 4 * d);
  const double c = (double)(p2 - p0);
  *dx = 3.0 * a * x * x + 2.0 * b * x + c;
  return __fma_rn(2.0, (double)p1, a * x2 * x + b * x2 + c * x);
}

// cubic1 with its multiplications by 2 and 1/2 folded: they are exact, so a
// fused multiply-add by them rounds once, where the addition does.
__device__ __forceinline__ double cubic1_fast(double p0, double p1, double p2, double p3, double x) {
  const double t0 = p2 - p0, t1 = p3 - p1;  // 2 fp0, 2 fp1
  const double c = 0.5 * t0;
  const double b = __fma_rn(-0.5, t1, 3.0 * p2 - 3.0 * p1 - t0);
  const double a = __fma_rn(0.5, t1, __fma_rn(2.0, p1 - p2, c));
  const double x2 = x * x;
  return a * x2 * x + b * x2 + c * x + p1;
}

}  // namespace ptk
