// fp64_ops.cuh -- scalar FP64 operations on the critical paths of the samplers, the register inverse and the
// Cholesky, and the FP64 matrix product of a warp.
//
// CUDA's double division, reciprocal and square root are calls of some 300 cycles; a proposal or an elimination step has
// several of them one after another.  The forms below start from the hardware's approximation (PTX rcp.approx and
// rsqrt.approx, about 20 bits), take three Newton steps and correct by the residual, which fma gives exactly.  Where
// an exponent is so extreme that a step could overflow or lose its residual, they call CUDA's operation.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// a / b from y, an approximation of 1 / b: the quotient a y and one residual correction (Markstein 1990), which is
// the rounded quotient when y is the rounded reciprocal and no exponent is extreme.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-q, b, a), y, q);
}

// 2^-e <= |v| < 2^e, by the exponent's bits (an integer test: an FP64 comparison would lengthen the chains it guards)
__device__ __forceinline__ bool moderate(double v, unsigned e) {
  const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
  return h - ((1023u - e) << 20) < (2u * e) << 20;
}

// 1 / b: the rounded reciprocal, but for a b whose significand is all ones (one unit in the last place).  b = 0,
// infinite, NaN or extreme: the division.
__device__ __forceinline__ double recip(double b) {
  if (!moderate(b, 930)) return 1.0 / b;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = fma(y, fma(-b, y, 1.0), y);
  y = fma(y, fma(-b, y, 1.0), y);
  return fma(y, fma(-b, y, 1.0), y);
}

// a / b for any a and b, with y = recip(b).  Where b or the quotient is extreme the correction may have overflowed or
// lost its residual (an infinite a y, for one, turns it into NaN): there the division.
__device__ __forceinline__ double quotient(double a, double b, double y) {
  const double q = div_by(a, b, y);
  return moderate(q, 100) && moderate(b, 830) ? q : __ddiv_rn(a, b);
}

// sqrt(d) and r = 1 / sqrt(d), each within one unit in the last place (d = 0, infinite, NaN or extreme: CUDA's)
__device__ __forceinline__ double sqrt_recip(double d, double& r) {
  if (!moderate(d, 930)) {
    r = rsqrt(d);
    return sqrt(d);
  }
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double h = 0.5 * d;
#pragma unroll
  for (int i = 0; i < 3; i++) y = fma(y, fma(-h * y, y, 0.5), y);
  r = y;
  const double s = d * y;
  return fma(fma(-s, s, d), 0.5 * y, s);
}

// y / (2^32 - 1) rounded (grnd, mt.f:70-102): equal to the division for every 32-bit y
__device__ __forceinline__ double word_fraction(uint32_t y) {
  return div_by((double)y, 4294967295.0, 1.0 / 4294967295.0);
}

// c += A B on the FP64 matrix units, 8 x 8 by one warp over four k: lane (g, t) = (lane / 4, lane % 4) gives A(g, t)
// and B(t, g) and holds c[e] = C(g, 2 t + e)
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
