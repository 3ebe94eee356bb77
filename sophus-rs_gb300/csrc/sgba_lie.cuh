// sgba_lie.cuh -- SE(3) in f64 on the device, with the derivative of the log
// along one direction, for cost terms on the poses themselves (pose priors and
// pose-graph edges).  Restates sophus_lie's unit-quaternion rotation and its
// affine group:
//   Rotation3 multiplication, matrix, log, mat_v_inverse and the w >= 0
//   disambiguation (crates/sophus_lie/src/groups/rotation3.rs:176-182,
//   389-410, 449-492, 778-800; crates/sophus_lie/src/lie_group/quaternion.rs);
//   the affine group's multiplication, inverse and log
//   (crates/sophus_lie/src/groups/affine_group_template.rs:362-404).
// Parameters (qw qx qy qz tx ty tz); tangent (w, v), rotation first.  An FP64
// instruction takes a warp 64 cycles whatever its lanes, so the forms are those
// with the fewest operations: rotations by two cross products, V^-1 t without
// its matrix.
#pragma once

#include <cuda_runtime.h>

namespace sgba {
namespace lie {

constexpr double kLieEps = 1e-6;  // EPS_F64 (crates/sophus_autodiff/src/linalg.rs:75)

__device__ __forceinline__ void cross(const double* a, const double* b, double* o) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

// Hamilton product: real a0 b0 - a_v . b_v, imaginary b_v a0 + a_v b0 + a_v x b_v
__device__ __forceinline__ void quat_mul(const double* a, const double* b, double* o) {
  o[0] = a[0] * b[0] - (a[1] * b[1] + a[2] * b[2] + a[3] * b[3]);
  o[1] = b[1] * a[0] + a[1] * b[0] + (a[2] * b[3] - a[3] * b[2]);
  o[2] = b[2] * a[0] + a[2] * b[0] + (a[3] * b[1] - a[1] * b[3]);
  o[3] = b[3] * a[0] + a[3] * b[0] + (a[1] * b[2] - a[2] * b[1]);
}

// rotation matrix of a unit quaternion, row-major
__device__ __forceinline__ void quat_matrix(const double* q, double* m) {
  const double x2 = 2.0 * q[1], y2 = 2.0 * q[2], z2 = 2.0 * q[3], r2 = 2.0 * q[0];
  const double xx = x2 * q[1], yy = y2 * q[2], zz = z2 * q[3];
  const double xy = x2 * q[2], xz = x2 * q[3], yz = y2 * q[3];
  const double rx = r2 * q[1], ry = r2 * q[2], rz = r2 * q[3];
  m[0] = 1.0 - (yy + zz);
  m[1] = xy - rz;
  m[2] = xz + ry;
  m[3] = xy + rz;
  m[4] = 1.0 - (xx + zz);
  m[5] = yz - rx;
  m[6] = xz - ry;
  m[7] = yz + rx;
  m[8] = 1.0 - (xx + yy);
}

// R(q) t = t + 2 (q0 (q_v x t) + q_v x (q_v x t))
__device__ __forceinline__ void rotate(const double* q, const double* t, double* o) {
  double c[3], e[3];
  cross(q + 1, t, c);
  cross(q + 1, c, e);
#pragma unroll
  for (int i = 0; i < 3; ++i) o[i] = t[i] + 2.0 * (q[0] * c[i] + e[i]);
}

// keep the real part non-negative; true if the signs were turned
__device__ __forceinline__ bool quat_disambiguate(double* q) {
  if (0.0 <= q[0]) return false;
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = -q[i];
  return true;
}

// a * b; true if the product quaternion's signs were turned
__device__ __forceinline__ bool se3_mul(const double* a, const double* b, double* o) {
  rotate(a, b + 4, o + 4);
#pragma unroll
  for (int i = 0; i < 3; ++i) o[4 + i] += a[4 + i];
  quat_mul(a, b, o);
  return quat_disambiguate(o);
}

// a^-1: conjugate rotation, -R^T t
__device__ __forceinline__ void se3_inverse(const double* a, double* o) {
  o[0] = a[0];
#pragma unroll
  for (int i = 1; i < 4; ++i) o[i] = -a[i];
  double t[3];
  rotate(o, a + 4, t);
#pragma unroll
  for (int i = 0; i < 3; ++i) o[4 + i] = -t[i];
  quat_disambiguate(o);
}

// log of (q, t): (w, V(w)^-1 t), and its derivative d along (dq, dt).
// w = f q_v: f = 2 atan(|q_v| / q_w) / |q_v|, or the series
// 2 / q_w - (2/3) |q_v|^2 / q_w^3 for |q_v|^2 <= eps^2.
// V(w)^-1 t = t - w x t / 2 + c w x (w x t), c = (1 - h cot h) / theta^2 with
// h = theta / 2 (1/12 for theta^2 <= eps); h cot h = f q_w / 2.
__device__ __forceinline__ void se3_log(const double* a, const double* dq, const double* dt, double* xi, double* d) {
  const double qw = a[0], dqw = dq[0];
  const double sq = a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
  const double hsq = a[1] * dq[1] + a[2] * dq[2] + a[3] * dq[3];  // half its derivative
  double f, df;
  if (sq <= kLieEps * kLieEps) {
    const double iw = 1.0 / qw, iw3 = iw * iw * iw;
    f = 2.0 * iw - (2.0 / 3.0) * sq * iw3;
    df = -2.0 * dqw * iw * iw - (4.0 / 3.0) * hsq * iw3 + 2.0 * sq * dqw * iw3 * iw;
  } else {
    const double n = sqrt(sq), in = 1.0 / n;
    const double sign = qw <= 0.0 ? -1.0 : 1.0;
    f = 2.0 * (sign * atan2(n, sign * qw)) * in;
    const double dn = hsq * in;
    df = (2.0 * (qw * dn - n * dqw) / (sq + qw * qw) - f * dn) * in;
  }
  const double* t = a + 4;
  double w[3], dw[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    w[i] = a[1 + i] * f;
    dw[i] = dq[1 + i] * f + a[1 + i] * df;
  }
  const double th2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
  double c = 1.0 / 12.0, dc = 0.0;
  if (th2 > kLieEps) {
    const double i2 = 1.0 / th2;
    c = (1.0 - 0.5 * f * qw) * i2;
    dc = -(0.5 * (df * qw + f * dqw) + 2.0 * c * (w[0] * dw[0] + w[1] * dw[1] + w[2] * dw[2])) * i2;
  }
  double y[3], z[3], p[3], r[3], dy[3];
  cross(w, t, y);
  cross(w, y, z);
  cross(dw, t, p);
  cross(w, dt, r);
#pragma unroll
  for (int i = 0; i < 3; ++i) dy[i] = p[i] + r[i];
  cross(dw, y, p);
  cross(w, dy, r);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    xi[i] = w[i];
    d[i] = dw[i];
    xi[3 + i] = t[i] - 0.5 * y[i] + c * z[i];
    d[3 + i] = dt[i] - 0.5 * dy[i] + (dc * z[i] + c * (p[i] + r[i]));
  }
}

}  // namespace lie
}  // namespace sgba
