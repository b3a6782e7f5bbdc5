// FP64 arithmetic from an FP32 seed, for the two places where a short chain of FP64 instructions is
// all that a kernel waits for: a Cholesky pivot's reciprocal and a Jacobi rotation. GB300's FP64
// pipe holds a warp's instruction for 64 cycles on a quarter of an SM, so the seeds and the
// conversions are integer and FP32 work.
//
// Both refinements are one step of Chebyshev's third-order method (J. F. Traub, Iterative Methods for
// the Solution of Equations, 1964), y + y (r + r^2) for 1/m with r = 1 - m y and
// y + y (e/2 + 3 e^2/8) for 1/sqrt(u) with e = 1 - u y^2: a seed good to 2^-21 leaves r^3, below
// 2^-62, and so the rounding of the last operations.
#pragma once
#include <cuda_runtime.h>

namespace gc {

// FP32 values from FP64 ones scaled by a common power of two (the larger exponent emax goes
// to 0), and back, by integer operations: conversions share the FP64 pipe.
__device__ __forceinline__ float to_scaled_f32(double x, int emax) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ff) - emax + 127;
  if (e < 1) return 0.f;
  return __uint_as_float((hi & 0x80000000u) | ((unsigned)e << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
}
__device__ __forceinline__ double f32_to_f64(float x) {  // x normal or zero
  const unsigned b = __float_as_uint(x);
  if ((b & 0x7f800000u) == 0) return 0.0;
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// 1 / d for d > 0, within one unit in the last place of the rounded quotient: the seed is the FP32
// reciprocal of the mantissa. A library square root and division are a chain of some 25 FP64
// instructions.
__device__ __forceinline__ double reciprocal(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const int e = (int)(hi >> 20) - 1023;  // d > 0
  if (e < -1000 || e > 1000) return 1.0 / d;
  const double m = __hiloint2double((int)((hi & 0xfffffu) | 0x3ff00000u), (int)lo);  // [1, 2)
  const float mf = __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29));
  const double y = f32_to_f64(__fdividef(1.f, mf));  // (1/2, 1]
  const double r = fma(-m, y, 1.0);
  const double z = fma(y, fma(r, r, r), y);
  return __hiloint2double((int)((unsigned)__double2hiint(z) - ((unsigned)e << 20)), __double2loint(z));
}

// The rotation (c, s) that takes the off-diagonal element h of a symmetric pair with the diagonal
// difference d = a_qq - a_pp away, tan = 2 h / (d +- sqrt(d^2 + 4 h^2)), in eight FP64 instructions
// (h not zero). The tangent is formed in FP32: it decides only how far h shrinks (to 1e-6 of
// itself); the rotation itself is orthogonal to FP64 rounding.
__device__ __forceinline__ void jacobi_rotation(double h, double d, double *c, double *s) {
  const int ed = (__double2hiint(d) >> 20) & 0x7ff, eh = (__double2hiint(h) >> 20) & 0x7ff;
  const int emax = max(ed, eh);
  const float df = to_scaled_f32(d, emax), hf = 2.f * to_scaled_f32(h, emax);
  const float r = sqrtf(df * df + hf * hf);
  const float tf = hf / (df >= 0.f ? df + r : df - r);
  const double t = f32_to_f64(tf), u = fma(t, t, 1.0);
  const double y = f32_to_f64(rsqrtf(fmaf(tf, tf, 1.f)));
  const double e = fma(-u, y * y, 1.0);
  *c = fma(e * y, fma(0.375, e, 0.5), y);
  *s = t * *c;
}

}  // namespace gc
