// pivot.cuh -- pivot arithmetic of the multifrontal factorisations.
//
// A GB300 sub-core issues one FP64 instruction per 64 cycles, whatever its
// active lanes, so what a pivot needs beside its multiply-subtracts is kept off
// that pipe or short.
#pragma once

namespace fgpu {

// 1 / d.  FP64: the hardware's approximate reciprocal and one third-order Newton
// step (e = 1 - d r; r (1 + e + e^2)), three multiply-adds on the critical chain
// in place of the division's five; the division itself outside the normal range.
__device__ inline float recip(float d) { return 1.0f / d; }
__device__ inline double recip(double d) {
  const unsigned ex = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
  if (ex - 64u > 1918u) return 1.0 / d;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  const double t = fma(e, e, e);
  return fma(r, t, r);
}
// v / d: the product with the reciprocal and one correction by its remainder
__device__ inline float quotient(float v, float d) { return v / d; }
__device__ inline double quotient(double v, double d) {
  const double r = recip(d), q = v * r;
  return fma(fma(-d, q, v), r, q);
}
// tests on the bit patterns of |x| (the order of non-negative patterns is the
// numeric order): they keep the FP64 pipe, one instruction per 64 cycles, free
__device__ inline bool absGreater(double a, double b) {
  const long long m = 0x7fffffffffffffffll;
  const long long x = __double_as_longlong(a) & m, y = __double_as_longlong(b) & m;
  return x > y && x <= 0x7ff0000000000000ll;
}
__device__ inline bool absGreater(float a, float b) { return fabsf(a) > fabsf(b); }
__device__ inline bool negative(double a) {
  const long long b = __double_as_longlong(a), m = b & 0x7fffffffffffffffll;
  return b < 0 && m != 0 && m <= 0x7ff0000000000000ll;
}
__device__ inline bool negative(float a) { return a < 0.0f; }
// the bound |d_k| must exceed for pivot k to count as regular
__device__ inline float singularBound(float a, float tol) { return tol * fabsf(a); }
__device__ inline double singularBound(double a, double tol) { return tol * fabs(a); }

}  // namespace fgpu
