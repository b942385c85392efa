// rotation.cuh -- 3x4 position matrices and finite rotations on the device,
// shared by the element, increment and joint kernels.
#pragma once

namespace fgpu {

// 3x4 position matrices, column-major: T[r + 3c]; o = a o b
__device__ inline void compose34(const double* a, const double* b, double* o) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double s = a[r] * b[3 * c] + a[r + 3] * b[3 * c + 1] + a[r + 6] * b[3 * c + 2];
      if (c == 3) s += a[r + 9];
      o[r + 3 * c] = s;
    }
}

__device__ inline void crossd(const double* a, const double* b, double* c) {
  double x = a[1] * b[2] - a[2] * b[1], y = a[2] * b[0] - a[0] * b[2], z = a[0] * b[1] - a[1] * b[0];
  c[0] = x; c[1] = y; c[2] = z;
}

// rotation tensor (column-major 3x3) of the unit quaternion q: 17 FP64 instructions,
// the products with 2 q shared between mirrored entries
__device__ inline void quatToMat(double q0, double q1, double q2, double q3, double* R) {
  const double p0 = q0 + q0, p1 = q1 + q1, p2 = q2 + q2, p3 = q3 + q3;
  const double w = fma(p0, q0, -1.0);
  const double a12 = p1 * q2, a13 = p1 * q3, a23 = p2 * q3;
  R[0] = fma(p1, q1, w);
  R[4] = fma(p2, q2, w);
  R[8] = fma(p3, q3, w);
  R[3] = fma(-p3, q0, a12);
  R[1] = fma(p3, q0, a12);
  R[6] = fma(p2, q0, a13);
  R[2] = fma(-p2, q0, a13);
  R[7] = fma(-p1, q0, a23);
  R[5] = fma(p1, q0, a23);
}

// rotation tensor from a rotation vector through a unit quaternion
// (rotationModule.f90:355-370,393-436).  For half angles below epsTh2 = 5e-4
// the reference interpolates sin(h)/h linearly (sinEpsOverEps = sin(epsTh2)/epsTh2,
// evaluated on the host); cos(h) is then its Taylor series to h^6 (the next
// term is below 1e-30), which spares the FP64 sine/cosine on the usual small
// increments.  The quaternion's squared norm is within 3e-14 of one in either case
// (the interpolation is off by at most 4e-8 in sin(h)/h, times h^2), so it is
// normalised by the first term of the reciprocal root's series, whose next is
// below 1e-27, in place of two reciprocal square roots.
__device__ inline void rotvecToMat(const double* rv, double sinEpsOverEps, double* R /* col-major 3x3 */) {
  const double epsTh2 = 0.0005;
  const double h2 = 0.25 * (rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
  double cthh, fac;
  if (h2 < epsTh2 * epsTh2) {
    cthh = 1.0 - h2 * (0.5 - h2 * (1.0 / 24.0 - h2 * (1.0 / 720.0)));
    // f1 = h / eps; it weighs 1 - sin(eps)/eps = 4e-8, so h = h2 rsqrt(h2) and the
    // product with 1 / eps (in place of a root and a division) do not show
    const double f1 = (h2 > 0.0 ? h2 * rsqrt(h2) : 0.0) * (1.0 / epsTh2);
    fac = f1 * sinEpsOverEps + 1.0 - f1;
  } else {
    const double thh = sqrt(h2);
    double sthh;
    sincos(thh, &sthh, &cthh);
    fac = sthh / thh;
  }
  fac *= 0.5;
  const double q1 = rv[0] * fac, q2 = rv[1] * fac, q3 = rv[2] * fac;
  const double inv = fma(-0.5, cthh * cthh + q1 * q1 + q2 * q2 + q3 * q3, 1.5);
  quatToMat(cthh * inv, q1 * inv, q2 * inv, q3 * inv, R);
}

}  // namespace fgpu
