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
// f / d for the multipliers of a pivot (0 when bad), as f r (1 + e + e^2) with the
// product f r beside the reciprocal's own Newton step: one multiply-add less on the
// pivot's critical chain than through recip(d)
struct PivotScale32 {
  float inv;
  __device__ PivotScale32(float d, bool bad) : inv(bad ? 0.0f : recip(d)) {}
  __device__ float operator()(float f) const { return f * inv; }
};
struct PivotScale64 {
  double r, t;
  __device__ PivotScale64(double d, bool bad) {
    const unsigned ex = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
    if (bad) {
      r = t = 0.0;
    } else if (ex - 64u > 1918u) {
      r = 1.0 / d;
      t = 0.0;
    } else {
      asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
      const double e = fma(-d, r, 1.0);
      t = fma(e, e, e);
    }
  }
  __device__ double operator()(double f) const {
    const double q = f * r;
    return fma(q, t, q);
  }
};
template <typename T> struct PivotScaleOf { using type = PivotScale32; };
template <> struct PivotScaleOf<double> { using type = PivotScale64; };
// v / d: the product with the reciprocal and one correction by its remainder
__device__ inline float quotient(float v, float d) { return v / d; }
__device__ inline double quotient(double v, double d) {
  const double r = recip(d), q = v * r;
  return fma(fma(-d, q, v), r, q);
}
// |x| as a bit pattern: for non-negative doubles the order of the patterns is the
// numeric order (NaN patterns are above infinity), so maxima and tests on it keep the
// FP64 pipe, one instruction per 64 cycles, free.  The sign is cleared on the high
// half: an AND on the 64-bit pattern is compiled into a floating-point absolute
// value, an FP64 instruction again.
__device__ __forceinline__ unsigned long long absBits(double x) {
  unsigned long long b;
  asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tand.b32 hi, hi, 0x7fffffff;\n\tmov.b64 %0, {lo, hi};\n\t}"
      : "=l"(b) : "d"(x));
  return b;
}
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;
__device__ inline bool absGreater(double a, double b) {
  const unsigned long long x = absBits(a), y = absBits(b);
  return x > y && x <= kInfBits;
}
__device__ inline bool absGreater(float a, float b) { return fabsf(a) > fabsf(b); }
__device__ inline bool negative(double a) {
  const unsigned long long m = absBits(a);
  return __double2hiint(a) < 0 && m != 0 && m <= kInfBits;
}
__device__ inline bool negative(float a) { return a < 0.0f; }
// the bound |d_k| must exceed for pivot k to count as regular
__device__ inline float singularBound(float a, float tol) { return tol * fabsf(a); }
__device__ inline double singularBound(double a, double tol) { return tol * fabs(a); }

}  // namespace fgpu
