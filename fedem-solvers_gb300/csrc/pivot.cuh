// pivot.cuh -- pivot arithmetic of the multifrontal factorisations.
//
// A GB300 sub-core issues one FP64 instruction per 64 cycles, whatever its
// active lanes, so what a pivot needs beside its multiply-subtracts is kept off
// that pipe or short.
#pragma once

namespace fgpu {

// |x| as a bit pattern: for non-negative doubles the order of the patterns is the
// numeric order (NaN patterns are above infinity), so maxima and tests on it keep the
// FP64 pipe, one instruction per 64 cycles, free.  The sign is cleared on the high
// 32-bit half (the norms' launch on 256 chains: 33 us with an AND on the 64-bit
// pattern, 27 us so).
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
