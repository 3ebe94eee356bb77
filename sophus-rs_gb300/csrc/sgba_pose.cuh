// sgba_pose.cuh -- SE(3) in f64 (restated from sophus_lie): the pose tables and
// the left-perturbation update of a pose by sixteen lanes.
#pragma once

#include <cuda_runtime.h>

#include "sgba_dd.cuh"

namespace {

constexpr double kPoseEps = 1e-6;  // EPS_F64 (crates/sophus_autodiff/src/linalg.rs:75)

// Rotation3Impl::matrix (crates/sophus_lie/src/groups/rotation3.rs:449-492)
__device__ void rot_matrix(const double* q, double* m) {
  double r = q[0], x = q[1], y = q[2], z = q[3];
  double tx = 2.0 * x, ty = 2.0 * y, tz = 2.0 * z, tr = 2.0 * r;
  double txx = tx * x, tyy = ty * y, tzz = tz * z;
  double txy = tx * y, txz = tx * z, tyz = ty * z;
  double trx = tr * x, try_ = tr * y, trz = tr * z;
  m[0] = 1.0 - (tyy + tzz); m[1] = txy - trz; m[2] = txz + try_;
  m[3] = txy + trz; m[4] = 1.0 - (txx + tzz); m[5] = tyz - trx;
  m[6] = txz - try_; m[7] = tyz + trx; m[8] = 1.0 - (txx + tyy);
}

// Pose tables: T_cw = T_wc^-1 in f64, published as float and float-float.
__device__ __forceinline__ void pose_table(const double* T, float* pf, float* pd) {
  double qc[4] = {T[0], -T[1], -T[2], -T[3]};
  double R[9];
  rot_matrix(qc, R);
  double t[3];
  for (int i = 0; i < 3; ++i) t[i] = -(R[i * 3 + 0] * T[4] + R[i * 3 + 1] * T[5] + R[i * 3 + 2] * T[6]);
  for (int i = 0; i < 12; ++i) {
    const dd v = dd_from_double(i < 9 ? R[i] : t[i - 9]);
    pf[i] = v.hi;
    pd[2 * i] = v.hi;
    pd[2 * i + 1] = v.lo;
  }
}

// --- the same by sixteen lanes -----------------------------------------------
// A warp's FP64 instruction takes its sub-partition 64 cycles whatever the
// number of active lanes, so one pose in one thread is bound by the count of
// its FP64 operations (~170 of them, and two sincos, two square roots, three
// divisions).  Here the entries of each small matrix, the two angles and the
// three divisions lie in lanes.  Which product of a sum is fused and which is
// rounded first is spelled out, and is this function's own definition; it was
// settled by comparing outputs with one thread's plain expressions, which the
// tables have to match: pose_table forms them from the same pose at the next
// linearisation, and a last-place change of a pose flips FP32 roundings there.
__device__ __forceinline__ double pose_neg(double x, bool n) {
  return n ? __longlong_as_double(__double_as_longlong(x) ^ (1ll << 63)) : x;
}
__device__ __forceinline__ double pose_pick(const double* v, int k) {  // v[k], k in 0 .. 3, v in registers
  const double a = (k & 1) ? v[1] : v[0], b = (k & 1) ? v[3] : v[2];
  return (k & 2) ? b : a;
}
__device__ __forceinline__ double pose_shfl(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane, 16); }

// Entry l (row-major, l < 9) of the rotation matrix of q; other lanes: unused.
__device__ __forceinline__ double rot_entry(const double* q, int l) {
  const int r = l / 3, c = l % 3;
  // diagonal: 1 - (t_u u + t_v v), u < v the other two axes; off it: t_a b +- t_r k,
  // a < b the entry's axes and k the third
  const bool diag = r == c;
  const int a = min(r, c) + 1, b = max(r, c) + 1;
  const int k = 6 - a - b;  // off the diagonal
  const int u = r == 0 ? 2 : 1, v = r == 2 ? 2 : 3;
  const double p0 = 2.0 * pose_pick(q, diag ? u : a), p1 = pose_pick(q, diag ? u : b);
  const double s0 = 2.0 * pose_pick(q, diag ? v : 0), s1 = pose_pick(q, diag ? v : k);
  // minus at (0,1), (1,2), (2,0)
  const bool minus = !diag && (c == r + 1 || (r == 2 && c == 0));
  // rot_matrix rounds one product on its own: the second, the first in (0,2) and
  // (2,0); in (0,0) both
  const bool first = l == 2 || l == 6;
  const double sn = pose_neg(s0, minus);
  const double fa = first ? sn : p0, fb = first ? s1 : p1, rest = (first ? p0 : sn) * (first ? p1 : s1);
  const double m = l == 0 ? __dadd_rn(__dmul_rn(fa, fb), rest) : fma(fa, fb, rest);
  return diag ? 1.0 - m : m;
}

// O = exp(xi) * T and its tables (Left-perturbation update
// crates/sophus_lie/src/lie_group/lie_group_manifold.rs:33-35,57-64;
//  exp: crates/sophus_lie/src/groups/affine_group_template.rs:354-360,
//       crates/sophus_lie/src/groups/rotation3.rs:363-387 and mat_v :761-778;
//  group_mul: affine_group_template.rs:387-396, quaternion.rs:212-225;
//  disambiguate: rotation3.rs:176-182) by the sixteen lanes of a half warp: lane l has xi[l] (l < 6) and T[l] (l < 7).
// The whole warp calls; lanes of a half that is `off` store nothing, those of a
// `still` one copy T.
__device__ __forceinline__ void pose_update16(double xil, double Tl, bool still, bool off, double* O, float* pf,
                                              float* pd) {
  const int l = threadIdx.x & 15;
  const int r = l / 3 % 3, c = l % 3;  // entry of lanes 0 .. 8
  double w[4], tr[3], T[7];
  for (int k = 0; k < 3; ++k) {
    w[k] = pose_shfl(xil, k);
    tr[k] = pose_shfl(xil, 3 + k);
  }
  w[3] = 0.0;
  for (int k = 0; k < 7; ++k) T[k] = pose_shfl(Tl, k);
  const double th2 = fma(w[2], w[2], fma(w[0], w[0], w[1] * w[1]));
  double eq[4];
  const bool small_q = th2 <= kPoseEps * kPoseEps, small_v = th2 <= kPoseEps;
  const double th = sqrt(th2);
  // lane 0: sin, cos of th / 2; lane 1: of th
  double s, co;
  sincos((l & 1) ? th : 0.5 * th, &s, &co);
  const double s0 = pose_shfl(s, 0), c0 = pose_shfl(co, 0), s1 = pose_shfl(s, 1), c1 = pose_shfl(co, 1);
  // lane 0: sin(th/2) / th; lane 1: (1 - cos th) / th^2; lane 2: (th - sin th) / th^3
  const double num = l == 0 ? s0 : (l == 1 ? 1.0 - c1 : th - s1);
  const double den = l == 0 ? th : (l == 1 ? th2 : th2 * th);
  const double quo = num / den;
  double im = pose_shfl(quo, 0);
  const double va = pose_shfl(quo, 1), vb = pose_shfl(quo, 2);
  eq[0] = c0;
  if (small_q) {
    const double th4 = th2 * th2;
    im = 0.5 - (1.0 / 48.0) * th2 + (1.0 / 3840.0) * th4;
    eq[0] = 1.0 - (1.0 / 8.0) * th2 + (1.0 / 384.0) * th4;
  }
  for (int k = 0; k < 3; ++k) eq[1 + k] = im * w[k];
  // mat_v = I + a W + b W^2 (0.5 W for small angles): entry (r, c)
  double et;
  {
    auto W = [&](int i, int j) {
      const double x = pose_pick(w, i == j ? 3 : 3 - i - j);
      return i == j ? 0.0 : pose_neg(x, j == i + 1 || (i == 2 && j == 0));
    };
    const double h = W(r, c);
    double v = 0.5 * h;
    if (!small_v) {
      double h2 = fma(W(r, 2), W(2, c), fma(W(r, 0), W(0, c), W(r, 1) * W(1, c)));
      if (l == 0) h2 = __dadd_rn(__dmul_rn(w[2], -w[2]), __dmul_rn(w[1], -w[1]));  // both products rounded
      if (l == 8) h2 = fma(w[0], -w[0], w[1] * -w[1]);
      v = fma(vb, h2, va * h);
    }
    if (r == c) v += 1.0;
    const int base = 3 * (l % 3);
    const double v0 = pose_shfl(v, base), v1 = pose_shfl(v, base + 1), v2 = pose_shfl(v, base + 2);
    // lanes 0 .. 2; v0 is the constant 1 in row 0 for small angles
    et = fma(v2, tr[2], (small_v && l == 0) ? fma(v1, tr[1], tr[0]) : fma(v0, tr[0], v1 * tr[1]));
  }
  if (!(0.0 <= eq[0]))
    for (int i = 0; i < 4; ++i) eq[i] = pose_neg(eq[i], true);
  // q = exp(xi)_q * T_q: lane 0 the real part, lanes 1 .. 3 the others
  double q[4];
  {
    const int i = l & 3, j = i == 3 ? 1 : i + 1, k = i == 1 ? 3 : i - 1;  // (i, j, k) cyclic for i = 1 .. 3
    double ql;
    if (i == 0) {
      ql = fma(eq[0], T[0], -fma(eq[3], T[3], fma(eq[1], T[1], eq[2] * T[2])));
    } else {
      const double cr = fma(pose_pick(eq, j), pose_pick(T, k), -(pose_pick(eq, k) * pose_pick(T, j)));
      ql = fma(pose_pick(T, i), eq[0], pose_pick(eq, i) * T[0]) + cr;
    }
    for (int n = 0; n < 4; ++n) q[n] = pose_shfl(ql, n);
  }
  const double R = rot_entry(eq, l);
  const int base = 3 * (l % 3);
  double ot;
  {
    const double r0 = pose_shfl(R, base), r1 = pose_shfl(R, base + 1), r2 = pose_shfl(R, base + 2);
    ot = fma(r2, T[6], fma(r0, T[4], r1 * T[5])) + et;  // lanes 0 .. 2: the translation
  }
  if (!(0.0 <= q[0]))
    for (int i = 0; i < 4; ++i) q[i] = pose_neg(q[i], true);
  double t[3];
  for (int k = 0; k < 3; ++k) t[k] = pose_shfl(ot, k);
  if (still) {
    for (int k = 0; k < 4; ++k) q[k] = T[k];
    for (int k = 0; k < 3; ++k) t[k] = T[4 + k];
  }
  if (!off && l < 7) O[l] = l < 4 ? pose_pick(q, l) : (l == 4 ? t[0] : (l == 5 ? t[1] : t[2]));
  // the tables of O
  for (int k = 1; k < 4; ++k) q[k] = pose_neg(q[k], true);
  const double Rc = rot_entry(q, l);
  const double r0 = pose_shfl(Rc, base), r1 = pose_shfl(Rc, base + 1), r2 = pose_shfl(Rc, base + 2);
  const double tc = pose_neg(fma(r2, t[2], fma(r0, t[0], r1 * t[1])), true);
  const double tcl = pose_shfl(tc, l >= 9 ? l - 9 : 0);
  if (!off && l < 12) {
    const dd v = dd_from_double(l < 9 ? Rc : tcl);
    pf[l] = v.hi;
    pd[2 * l] = v.hi;
    pd[2 * l + 1] = v.lo;
  }
}

}  // namespace
