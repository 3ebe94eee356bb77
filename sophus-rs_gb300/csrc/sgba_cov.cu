// sgba_cov.cu -- covariance and precision queries of the final Hessian on the
// GPU.
//
// Reference: Optimizer::build_solution (crates/sophus_opt/src/nlls/optimizer.rs:609-646)
// evaluates the linear system at the solution with zero damping;
// OptimizationSolution::precision_block / covariance_block
// (crates/sophus_opt/src/nlls/optimizer_types.rs:277-370) answer block queries
// from it.  The Schur factor answers covariance blocks as
// SchurFactor::inverse_block does (crates/sophus_solver/src/ldlt/schur_ldlt.rs:815-957):
//   free x free  S^-1[row, col]
//   free x marg  -(S^-1 H_fm H_mm^-1)[row, col]
//   marg x marg  H_mm^-1 delta_ij + H_mm[i]^-1 H_mf_i S^-1 H_mf_j^T H_mm[j]^-1
// and S^-1 is the min-norm pseudo-inverse E G^-1 diag(d_J)^-1 G^-1 E^T when
// the LDL^T of S has zero pivots (crates/sophus_solver/src/ldlt/min_norm_ldlt.rs:55-140),
// E the columns of L at the positive pivots J and G = E^T E.
//
// Arithmetic: f64 throughout (FP64 pipe).  The covariance inverts S, so its
// error is the error of S times the condition number of S; the LM path's
// FP32 / float-float linearization is accurate enough for a step that the
// next iteration corrects, not for an inverse.  The Hessian of a
// reprojection term is J^T J whatever the robust kernel (the weight acts on
// the residual), so only the Jacobians enter: they are evaluated here in f64
// from the same closed forms as the linearization kernels.
//
// Kernels, in order:
//   k_cov_groups     thread per reduced term (point, pose): J_pose^T J_pose,
//                    W = J_pose^T J_point, J_point^T J_point (times the
//                    term's observation count: its observations share J)
//   k_cov_points     thread per marginalized point: H_mm = sum over its terms
//                    (term order) and its inverse (cofactors, singular iff
//                    the determinant is 0, as nalgebra's try_inverse)
//   k_cov_y          Y = W H_mm^-1 of the terms with a free pose
//   k_cov_s          CTA per lower block (a, b) of S: the diagonal block
//                    U_a + priors + edges - sum Y W^T over pose a's terms;
//                    off-diagonal blocks - sum Y_a W_b^T over the points both
//                    poses see (32 slices of pose a's term list, in point
//                    order, searched in pose b's) + J_m^T J_n of edges;
//                    both triangles written.  No atomics: lane sums by a
//                    fixed shuffle tree, one writer per entry.
//   k_cov_diag /     right-looking scalar LDL^T in natural order, 6-row pose
//   k_cov_rows /     blocks with the reference's pivot rule
//   k_cov_update     (dense_ldlt.rs:164-230: a pivot at most
//                    1e-12 max(1, largest pivot so far in its block) is
//                    zeroed and zeroes its column of L), launched by panels
//                    of eight: the panel's diagonal block, the rows below it,
//                    the trailing lower triangle in 32 x 32 tiles
//   k_cov_winv /     S^-1 = W^T D^-1 W, W = L^-1 by doubling blocks, and the
//   k_cov_wlevel /   product
//   k_cov_wtw
//   k_cov_gemm       tiled f64 products of the pseudo-inverse (rank-deficient S)
//   k_cov_query      CTA per query: covariance or H blocks from Z, Y, H_mm^-1
#include <cuda_runtime.h>

#include <cfloat>
#include <algorithm>
#include <cstdint>
#include <vector>

#include "sgba_internal.h"
#include "sgba_lie.cuh"

namespace sgba {

namespace {

constexpr int kCovThreads = 256;
constexpr double kCovTolRel = 1e-12;  // BlockSparseLdlt's tol_rel
constexpr int kUT = 32;               // trailing-update tile
constexpr int kGT = 64, kGK = 16;     // GEMM tile and depth

// ---------------------------------------------------------------------------
// Jacobians of r = uv - pi(T_cw p) in f64 (the closed forms of the
// linearization kernels, pinhole_reprojection.rs:60-95, ba_problem.rs:69-110):
// T_cw = T_wc^-1, D = d pi R_cw (2x3), J_pose = [D hat(-p), D], J_point = -D.
// ---------------------------------------------------------------------------
template <bool E>
__device__ void cov_jacobians(const double* T, const double* p, const double* intr, double* jp, double* jm) {
  double Rwc[9];
  lie::quat_matrix(T, Rwc);
  double R[9], t[3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) R[3 * i + j] = Rwc[3 * j + i];
  for (int i = 0; i < 3; ++i) t[i] = -(R[3 * i] * T[4] + R[3 * i + 1] * T[5] + R[3 * i + 2] * T[6]);
  const double xc = R[0] * p[0] + R[1] * p[1] + R[2] * p[2] + t[0];
  const double yc = R[3] * p[0] + R[4] * p[1] + R[5] * p[2] + t[1];
  const double zc = R[6] * p[0] + R[7] * p[1] + R[8] * p[2] + t[2];
  const double iz = 1.0 / zc;
  const double fx = intr[0], fy = intr[1];
  double D[6];
  if constexpr (!E) {
    const double a0 = fx * iz, a2 = -fx * xc * iz * iz;
    const double b1 = fy * iz, b2 = -fy * yc * iz * iz;
    for (int k = 0; k < 3; ++k) {
      D[k] = a0 * R[k] + a2 * R[6 + k];
      D[3 + k] = b1 * R[3 + k] + b2 * R[6 + k];
    }
  } else {
    // d pi = M d proj, M the derivative of the EUCM distortion (enhanced_unified.rs:117-156)
    const double al = intr[4], be = intr[5];
    const double x = xc * iz, y = yc * iz;
    const double rho = sqrt(be * (x * x + y * y) + 1.0);
    const double nrm = al * rho + (1.0 - al);
    const double in2 = 1.0 / (nrm * nrm);
    const double ab = al * be / rho;
    const double nx = ab * x, ny = ab * y;
    const double m00 = fx * (nrm - x * nx) * in2, m01 = -fx * x * ny * in2;
    const double m10 = -fy * y * nx * in2, m11 = fy * (nrm - y * ny) * in2;
    const double a0 = m00 * iz, a1 = m01 * iz, a2 = -(m00 * x + m01 * y) * iz;
    const double b0 = m10 * iz, b1 = m11 * iz, b2 = -(m10 * x + m11 * y) * iz;
    for (int k = 0; k < 3; ++k) {
      D[k] = a0 * R[k] + a1 * R[3 + k] + a2 * R[6 + k];
      D[3 + k] = b0 * R[k] + b1 * R[3 + k] + b2 * R[6 + k];
    }
  }
  const double px = p[0], py = p[1], pz = p[2];
  for (int r = 0; r < 2; ++r) {
    const double* d = D + 3 * r;
    jp[r * 6 + 0] = -d[1] * pz + d[2] * py;
    jp[r * 6 + 1] = d[0] * pz - d[2] * px;
    jp[r * 6 + 2] = -d[0] * py + d[1] * px;
    jp[r * 6 + 3] = d[0];
    jp[r * 6 + 4] = d[1];
    jp[r * 6 + 5] = d[2];
    jm[r * 3 + 0] = -d[0];
    jm[r * 3 + 1] = -d[1];
    jm[r * 3 + 2] = -d[2];
  }
}

// index of (a, b), a <= b, in the row-major upper triangle of a k x k matrix
__device__ __forceinline__ int up_idx(int k, int a, int b) { return a * k - a * (a - 1) / 2 + (b - a); }

// Jacobian of r with respect to the camera params (2 x 6 row-major, columns
// beyond the model's 4 or 6 zero): J_cam = -d pi / d params
// (pinhole_reprojection.rs:85, dx_distort_params of perspective.rs and
// enhanced_unified.rs:158-215): fx fy cx cy, then for the EUCM camera
// alpha beta with d(1/norm) / d alpha = -(rho - 1) / norm^2 and
// d(1/norm) / d beta = -alpha r2 / (2 rho norm^2).
template <bool E>
__device__ void cov_cam_jacobian(const double* T, const double* p, const double* intr, double* jc) {
  double Rwc[9];
  lie::quat_matrix(T, Rwc);
  double R[9], t[3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) R[3 * i + j] = Rwc[3 * j + i];
  for (int i = 0; i < 3; ++i) t[i] = -(R[3 * i] * T[4] + R[3 * i + 1] * T[5] + R[3 * i + 2] * T[6]);
  const double xc = R[0] * p[0] + R[1] * p[1] + R[2] * p[2] + t[0];
  const double yc = R[3] * p[0] + R[4] * p[1] + R[5] * p[2] + t[1];
  const double zc = R[6] * p[0] + R[7] * p[1] + R[8] * p[2] + t[2];
  const double x = xc / zc, y = yc / zc;
  for (int k = 0; k < 12; ++k) jc[k] = 0.0;
  jc[2] = -1.0;
  jc[6 + 3] = -1.0;
  if constexpr (E) {
    const double al = intr[4], be = intr[5];
    const double r2 = x * x + y * y;
    const double rho = sqrt(be * r2 + 1.0);
    const double nrm = al * rho + (1.0 - al);
    const double in2 = 1.0 / (nrm * nrm);
    const double da = (rho - 1.0) * in2;
    const double db = al * r2 * in2 / (2.0 * rho);
    jc[0] = -x / nrm;
    jc[6 + 1] = -y / nrm;
    jc[4] = intr[0] * x * da;
    jc[5] = intr[0] * x * db;
    jc[6 + 4] = intr[1] * y * da;
    jc[6 + 5] = intr[1] * y * db;
  } else {
    jc[0] = -x;
    jc[6 + 1] = -y;
  }
}

template <bool E>
__global__ void __launch_bounds__(kCovThreads) k_cov_groups(int64_t ng, const int64_t* __restrict__ g_begin,
                                                           const int32_t* __restrict__ g_pose,
                                                           const int32_t* __restrict__ g_pt,
                                                           const double* __restrict__ poses,
                                                           const double* __restrict__ points,
                                                           const double* __restrict__ intr, double* __restrict__ rec,
                                                           double* __restrict__ crec) {
  const int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (g >= ng) return;
  double jp[12], jm[6];
  const double* T = poses + 7 * static_cast<int64_t>(g_pose[g]);
  const double* P = points + 3 * static_cast<int64_t>(g_pt[g]);
  cov_jacobians<E>(T, P, intr, jp, jm);
  const double cnt = static_cast<double>(g_begin[g + 1] - g_begin[g]);
  double* o = rec + kCovRec * g;
  int k = 0;
  for (int a = 0; a < 6; ++a)
    for (int b = a; b < 6; ++b) o[k++] = cnt * (jp[a] * jp[b] + jp[6 + a] * jp[6 + b]);
  for (int a = 0; a < 6; ++a)
    for (int j = 0; j < 3; ++j) o[21 + 3 * a + j] = cnt * (jp[a] * jm[j] + jp[6 + a] * jm[3 + j]);
  k = 39;
  for (int i = 0; i < 3; ++i)
    for (int j = i; j < 3; ++j) o[k++] = cnt * (jm[i] * jm[j] + jm[3 + i] * jm[3 + j]);
  if (!crec) return;
  // free camera params: J_cam^T J_cam (21 upper), J_cam^T J_pose (6 x 6), J_cam^T J_point (6 x 3)
  double jc[12];
  cov_cam_jacobian<E>(T, P, intr, jc);
  double* oc = crec + kCovCamRec * g;
  k = 0;
  for (int a = 0; a < 6; ++a)
    for (int b = a; b < 6; ++b) oc[k++] = cnt * (jc[a] * jc[b] + jc[6 + a] * jc[6 + b]);
  for (int a = 0; a < 6; ++a)
    for (int b = 0; b < 6; ++b) oc[21 + 6 * a + b] = cnt * (jc[a] * jp[b] + jc[6 + a] * jp[6 + b]);
  for (int a = 0; a < 6; ++a)
    for (int j = 0; j < 3; ++j) oc[57 + 3 * a + j] = cnt * (jc[a] * jm[j] + jc[6 + a] * jm[3 + j]);
}

// nalgebra's 3x3 try_inverse: adjugate / determinant, singular iff det == 0
__device__ bool inverse3(const double* m, double* o) {
  const double m11 = m[0], m12 = m[1], m13 = m[2];
  const double m21 = m[3], m22 = m[4], m23 = m[5];
  const double m31 = m[6], m32 = m[7], m33 = m[8];
  const double c11 = m22 * m33 - m32 * m23;
  const double c21 = m21 * m33 - m31 * m23;
  const double c31 = m21 * m32 - m31 * m22;
  const double det = m11 * c11 - m12 * c21 + m13 * c31;
  if (det == 0.0) return false;
  o[0] = c11 / det;
  o[1] = (m13 * m32 - m33 * m12) / det;
  o[2] = (m12 * m23 - m22 * m13) / det;
  o[3] = -c21 / det;
  o[4] = (m11 * m33 - m31 * m13) / det;
  o[5] = (m13 * m21 - m23 * m11) / det;
  o[6] = c31 / det;
  o[7] = (m12 * m31 - m32 * m11) / det;
  o[8] = (m11 * m22 - m21 * m12) / det;
  return true;
}

// A thread per point: H_mm over the point's terms in order and its inverse.
constexpr int kCovPtT = 64;  // small CTAs: a few thousand points spread over the GPU
__global__ void __launch_bounds__(kCovPtT) k_cov_points(int np, const int64_t* __restrict__ pt_g_begin,
                                                       const int32_t* __restrict__ pt_mb,
                                                       const double* __restrict__ rec, double* __restrict__ vinv,
                                                       int* status, const double* __restrict__ crec,
                                                       double* __restrict__ wc, double* __restrict__ yc) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= np) return;
  const int mb = pt_mb[q];
  if (mb < 0) return;
  double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 4
  for (int64_t g = pt_g_begin[q]; g < pt_g_begin[q + 1]; ++g)
    for (int k = 0; k < 6; ++k) v[k] += rec[kCovRec * g + 39 + k];
  const double V[9] = {v[0], v[1], v[2], v[1], v[3], v[4], v[2], v[4], v[5]};
  double Vi[9];
  double* vo = vinv + 9 * static_cast<int64_t>(mb);
  if (!inverse3(V, Vi)) {
    for (int k = 0; k < 9; ++k) vo[k] = __longlong_as_double(0x7ff8000000000000ll);
    atomicOr(status + 1, 1);
    return;
  }
  for (int k = 0; k < 9; ++k) vo[k] = Vi[k];
  if (!crec) return;
  // free camera params: W_cq = sum of the point's J_cam^T J_point, Y_cq = W_cq H_mm^-1
  double W[18];
  for (int k = 0; k < 18; ++k) W[k] = 0.0;
  for (int64_t g = pt_g_begin[q]; g < pt_g_begin[q + 1]; ++g)
    for (int k = 0; k < 18; ++k) W[k] += crec[kCovCamRec * g + 57 + k];
  double* wo = wc + 18 * static_cast<int64_t>(mb);
  double* yo = yc + 18 * static_cast<int64_t>(mb);
  for (int a = 0; a < 6; ++a)
    for (int j = 0; j < 3; ++j) {
      wo[3 * a + j] = W[3 * a + j];
      yo[3 * a + j] = W[3 * a] * Vi[j] + W[3 * a + 1] * Vi[3 + j] + W[3 * a + 2] * Vi[6 + j];
    }
}

// Y = W H_mm^-1 of the terms with a free pose and a marginalized point (zero
// for the others), a thread per row.  (The thread per point that formed them
// term by term left most of the GPU idle: 188 us for 5,001 points of 25 terms.)
__global__ void __launch_bounds__(kCovThreads) k_cov_y(int64_t ng, const int32_t* __restrict__ g_pose,
                                                      const int32_t* __restrict__ g_pt,
                                                      const int32_t* __restrict__ pose_fb,
                                                      const int32_t* __restrict__ pt_mb,
                                                      const double* __restrict__ rec,
                                                      const double* __restrict__ vinv, double* __restrict__ y) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t g = e / 6;
  if (g >= ng) return;
  const int a = static_cast<int>(e - 6 * g);
  const int mb = pt_mb[g_pt[g]];
  double* yo = y + 18 * g + 3 * a;
  if (mb < 0 || pose_fb[g_pose[g]] < 0) {
    for (int j = 0; j < 3; ++j) yo[j] = 0.0;
    return;
  }
  const double* W = rec + kCovRec * g + 21;
  const double* Vi = vinv + 9 * static_cast<int64_t>(mb);
#pragma unroll
  for (int j = 0; j < 3; ++j) yo[j] = W[3 * a] * Vi[j] + W[3 * a + 1] * Vi[3 + j] + W[3 * a + 2] * Vi[6 + j];
}

// The camera block of S (free camera params, rows 0..5 of S; rows nk..5 are
// padding: identity): H_cc = sum over every term of J_cam^T J_cam, minus
// sum over the marginalized points of Y_cq W_cq^T.  One CTA; thread t sums
// terms and points t, t + 256, ...; the threads' sums by a fixed tree.
__global__ void __launch_bounds__(kCovThreads) k_cov_cam(int64_t ng, int nm, int nk, int n,
                                                        const double* __restrict__ crec,
                                                        const double* __restrict__ wc, const double* __restrict__ yc,
                                                        double* __restrict__ S, double* __restrict__ hcc) {
  __shared__ double red[kCovThreads];
  double h[21], sc[21];
  for (int k = 0; k < 21; ++k) h[k] = sc[k] = 0.0;
  for (int64_t g = threadIdx.x; g < ng; g += blockDim.x)
    for (int k = 0; k < 21; ++k) h[k] += crec[kCovCamRec * g + k];
  for (int mb = threadIdx.x; mb < nm; mb += blockDim.x) {
    const double* W = wc + 18 * static_cast<int64_t>(mb);
    const double* Y = yc + 18 * static_cast<int64_t>(mb);
    int k = 0;
    for (int a = 0; a < 6; ++a)
      for (int b = a; b < 6; ++b, ++k) sc[k] += Y[3 * a] * W[3 * b] + Y[3 * a + 1] * W[3 * b + 1] + Y[3 * a + 2] * W[3 * b + 2];
  }
  for (int part = 0; part < 2; ++part)
    for (int k = 0; k < 21; ++k) {
      red[threadIdx.x] = part == 0 ? h[k] : sc[k];
      __syncthreads();
      for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
      }
      if (threadIdx.x == 0) {
        if (part == 0) h[k] = red[0];
        else sc[k] = red[0];
      }
      __syncthreads();
    }
  if (threadIdx.x != 0) return;
  for (int a = 0; a < 6; ++a)
    for (int b = 0; b < 6; ++b) {
      const int k = a <= b ? up_idx(6, a, b) : up_idx(6, b, a);
      const bool real = a < nk && b < nk;
      hcc[6 * a + b] = real ? h[k] : 0.0;
      S[static_cast<int64_t>(a) * n + b] = real ? h[k] - sc[k] : (a == b ? 1.0 : 0.0);
    }
}

struct CovSArgs {
  int64_t nsb;
  int n;
  const int32_t* sb_row;
  const int32_t* sb_col;
  const int64_t* fb_tile_begin;
  const int64_t* tile_begin;
  const int64_t* tile_end;
  const int64_t* cam_g;
  const int32_t* cam_pt;     // point of every entry of cam_g
  const int32_t* pt_mb;
  const double* rec;
  const double* y;
  const int32_t* prior_beg;  // per free block: its priors (null: none)
  const double* prior_out;
  const int32_t* e_beg;      // per free block: its edge records (null: none)
  const int32_t* e_slot;
  const double* e_out;
  const int32_t* eblk_begin;  // per lower block: its edge terms (bit 31: transposed)
  const int32_t* eblk_term;
  const double* e_hmn;
  double* S;
  double* hdiag;
  int nci;             // rows of the camera block before the poses (6 with free camera params, else 0)
  const double* crec;  // free camera params: per-term camera records (null: conditioned)
  const double* wc;    // per marginalized point W_cq (6 x 3)
  double* hcp;         // per free pose H_ca (camera rows x pose columns, 6 x 6)
};

// the term-list range of free pose fb (its camera tiles are contiguous in cam_g)
__device__ __forceinline__ void cam_range(const CovSArgs& a, int fb, int64_t* b, int64_t* e) {
  const int64_t t0 = a.fb_tile_begin[fb], t1 = a.fb_tile_begin[fb + 1];
  *b = t0 < t1 ? a.tile_begin[t0] : 0;
  *e = t0 < t1 ? a.tile_end[t1 - 1] : 0;
}

// row r of acc (6x6) -= Y W^T, Y the row's three entries
__device__ __forceinline__ void sub_ywt(double* acc, const double* Y, const double* W) {
#pragma unroll
  for (int c = 0; c < 6; ++c) acc[c] -= Y[0] * W[3 * c] + Y[1] * W[3 * c + 1] + Y[2] * W[3 * c + 2];
}

// the lanes' sums of a warp by a fixed shuffle tree (lane 0 holds the totals)
__device__ __forceinline__ void warp_sum6(double* acc) {
#pragma unroll
  for (int k = 0; k < 6; ++k)
    for (int off = 16; off > 0; off >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], off);
}

// the point of every entry of the cameras' term lists
__global__ void __launch_bounds__(kCovThreads) k_cov_cam_pt(int64_t n, const int64_t* __restrict__ cam_g,
                                                           const int32_t* __restrict__ g_pt, int32_t* __restrict__ out) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e < n) out[e] = g_pt[cam_g[e]];
}

// A CTA per lower block (fa, fb) of S, warp r its row r.  Diagonal blocks: the
// lanes take pose fa's terms in turn.  Off-diagonal blocks: lane l takes its
// slice of pose fa's term list (1/32 of it, in point order): for a piece of
// every slice the CTA first finds the terms of pose fb on the same points (a
// binary search per term, all of them at once), then the lanes add theirs in
// order (matches packed to the front of each slice: the FP64 pipe takes a step's
// time for one lane as for 32, and that pipe bounds this kernel, 77 % busy).  (A
// warp per block that merged the two lists step by step, 36 sums a
// lane, spent its time on the chain of list loads: 1.5 ms for 741 blocks of
// 1,250 x 1,250 terms.)
constexpr int kCovSThreads = 192;
constexpr int kCovPiece = 32;  // terms of a slice searched at once
constexpr int kCovStage = 8;   // of which this many have their W (6x3) in shared memory at a time
__global__ void __launch_bounds__(kCovSThreads) k_cov_s(CovSArgs a) {
  __shared__ int s_gi[kCovPiece][32], s_gj[kCovPiece][32];
  // W of the matches, [entry][match]: the lanes' own reads of 18 entries from 32
  // records would take 32 cache wavefronts each, for every row's warp
  __shared__ double s_w[18][kCovStage * 32];
  __shared__ int s_most;
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
  const int64_t s = blockIdx.x;
  const int fa = a.sb_row[s], fb = a.sb_col[s];
  double acc[6] = {0, 0, 0, 0, 0, 0};
  int64_t ib, ie;
  cam_range(a, fa, &ib, &ie);
  if (fa == fb) {
    for (int64_t i = ib + lane; i < ie; i += 32) {
      const double* h = a.rec + kCovRec * a.cam_g[i];
#pragma unroll
      for (int c = 0; c < 6; ++c) acc[c] += h[r <= c ? up_idx(6, r, c) : up_idx(6, c, r)];
    }
    warp_sum6(acc);
    if (lane == 0) {
      if (a.prior_beg)
        for (int q = a.prior_beg[fa]; q < a.prior_beg[fa + 1]; ++q)
          for (int c = 0; c < 6; ++c) acc[c] += a.prior_out[static_cast<int64_t>(kPriorOut) * q + 6 * r + c];
      if (a.e_beg)
        for (int q = a.e_beg[fa]; q < a.e_beg[fa + 1]; ++q)
          for (int c = 0; c < 6; ++c) acc[c] += a.e_out[static_cast<int64_t>(kPriorOut) * a.e_slot[q] + 6 * r + c];
      for (int c = 0; c < 6; ++c) a.hdiag[36 * static_cast<int64_t>(fa) + 6 * r + c] = acc[c];
    }
    // the Schur part, then lane 0 adds back the H block it stored
    double h0[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      h0[c] = acc[c];
      acc[c] = 0.0;
    }
    for (int64_t i = ib + lane; i < ie; i += 32) {
      const int64_t g = a.cam_g[i];
      if (a.pt_mb[a.cam_pt[i]] < 0) continue;
      sub_ywt(acc, a.y + 18 * g + 3 * r, a.rec + kCovRec * g + 21);
    }
    warp_sum6(acc);
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] += h0[c];
  } else {
    int64_t jb, je;
    cam_range(a, fb, &jb, &je);
    const int64_t len = ie - ib;
    const int64_t longest = (len + 31) / 32;
    for (int64_t p0 = 0; p0 < longest; p0 += kCovPiece) {
      __syncthreads();
#pragma unroll 2
      for (int e = threadIdx.x; e < 32 * kCovPiece; e += kCovSThreads) {
        const int l = e & 31, u = e >> 5;
        const int64_t i = ib + len * l / 32 + p0 + u;
        int gi = 0, gj = -1;
        if (i < ib + len * (l + 1) / 32) {
          const int pt = a.cam_pt[i];
          if (a.pt_mb[pt] >= 0) {
            int64_t lo = jb, hi = je;
            while (lo < hi) {
              const int64_t mid = lo + (hi - lo) / 2;
              if (a.cam_pt[mid] < pt) lo = mid + 1;
              else hi = mid;
            }
            if (lo < je && a.cam_pt[lo] == pt) {
              gi = static_cast<int>(a.cam_g[i]);
              gj = static_cast<int>(a.cam_g[lo]);
            }
          }
        }
        s_gi[u][l] = gi;
        s_gj[u][l] = gj;
      }
      __syncthreads();
      if (r == 0) {  // every lane's matches to the front of its slice, in order
        int m = 0;
        for (int u = 0; u < kCovPiece; ++u) {
          const int gi = s_gi[u][lane], gj = s_gj[u][lane];
          if (gj < 0) continue;
          s_gi[m][lane] = gi;
          s_gj[m][lane] = gj;
          ++m;
        }
        for (int u = m; u < kCovPiece; ++u) s_gj[u][lane] = -1;
        const int most = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) s_most = most;
      }
      __syncthreads();
      const int un = s_most;
      for (int u0 = 0; u0 < un; u0 += kCovStage) {
#pragma unroll 8
        for (int e = threadIdx.x; e < 18 * kCovStage * 32; e += kCovSThreads) {
          const int m = e / 18, k = e - 18 * m;
          const int gj = s_gj[u0 + (m >> 5)][m & 31];
          if (gj >= 0) s_w[k][m] = a.rec[kCovRec * static_cast<int64_t>(gj) + 21 + k];
        }
        __syncthreads();
        for (int u = 0; u < kCovStage && u0 + u < un; ++u) {
          if (s_gj[u0 + u][lane] < 0) continue;
          const double* Y = a.y + 18 * static_cast<int64_t>(s_gi[u0 + u][lane]) + 3 * r;
          const double y0 = Y[0], y1 = Y[1], y2 = Y[2];
          const int m = 32 * u + lane;
#pragma unroll
          for (int c = 0; c < 6; ++c) acc[c] -= y0 * s_w[3 * c][m] + y1 * s_w[3 * c + 1][m] + y2 * s_w[3 * c + 2][m];
        }
        __syncthreads();
      }
    }
    warp_sum6(acc);
    if (lane == 0 && a.eblk_begin)
      for (int q = a.eblk_begin[s]; q < a.eblk_begin[s + 1]; ++q) {
        const int32_t tt = a.eblk_term[q];
        const int64_t term = tt & 0x7fffffff;
        for (int c = 0; c < 6; ++c)
          acc[c] += (tt < 0) ? a.e_hmn[36 * term + c * 6 + r] : a.e_hmn[36 * term + r * 6 + c];
      }
  }
  const int64_t n = a.n;
  if (lane == 0)
    for (int c = 0; c < 6; ++c) {
      if (fa == fb && c > r) continue;  // the diagonal block from its lower triangle (exactly symmetric)
      const int64_t row = a.nci + 6 * fa + r, col = a.nci + 6 * fb + c;
      a.S[row * n + col] = acc[c];
      a.S[col * n + row] = acc[c];
    }
  if (fa != fb || !a.crec) return;
  // free camera params: the pose's camera columns S_ac = H_ac - sum over its
  // terms with a marginalized point of Y_g W_cq^T (acc[k]: pose row r, camera column k)
#pragma unroll
  for (int k = 0; k < 6; ++k) acc[k] = 0.0;
  for (int64_t i = ib + lane; i < ie; i += 32) {
    const double* hc = a.crec + kCovCamRec * a.cam_g[i] + 21;
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] += hc[6 * k + r];
  }
  warp_sum6(acc);
  double h0[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    h0[k] = acc[k];
    if (lane == 0) a.hcp[36 * static_cast<int64_t>(fa) + 6 * k + r] = acc[k];
    acc[k] = 0.0;
  }
  for (int64_t i = ib + lane; i < ie; i += 32) {
    const int64_t g = a.cam_g[i];
    const int mb = a.pt_mb[a.cam_pt[i]];
    if (mb < 0) continue;
    sub_ywt(acc, a.y + 18 * g + 3 * r, a.wc + 18 * static_cast<int64_t>(mb));
  }
  warp_sum6(acc);
  if (lane != 0) return;
  for (int k = 0; k < 6; ++k) {
    const double v = h0[k] + acc[k];
    const int64_t row = a.nci + 6 * fa + r;
    a.S[row * n + k] = v;
    a.S[static_cast<int64_t>(k) * n + row] = v;
  }
}

// ---------------------------------------------------------------------------
// LDL^T
// ---------------------------------------------------------------------------

// dense_ldlt.rs:164-230 on the 6x6 block a (row-major, lower used): unit-lower
// L in a, pivots in d.  Returns 0, 1 for a non-finite pivot, 2 for an
// indefinite block whose pivot condition is below the Bunch-Kaufman threshold.
__device__ int ldlt6(double* a, double* d) {
  double maxp = 1.0, minp = DBL_MAX;
  int rank = 0;
  bool neg = false;
  for (int j = 0; j < 6; ++j) {
    for (int k = 0; k < j; ++k) {
      double s = a[6 * j + k];
      for (int p = 0; p < k; ++p) s -= a[6 * j + p] * d[p] * a[6 * k + p];
      const double tol = fmax(maxp, 1.0) * kCovTolRel;
      a[6 * j + k] = (fabs(d[k]) <= tol) ? 0.0 : s / d[k];
    }
    double djj = a[6 * j + j];
    for (int p = 0; p < j; ++p) djj -= d[p] * a[6 * j + p] * a[6 * j + p];
    if (!isfinite(djj)) return 1;
    const double tol = fmax(maxp, 1.0) * kCovTolRel;
    if (fabs(djj) <= tol) {
      d[j] = 0.0;
    } else {
      if (djj < 0.0) neg = true;
      d[j] = djj;
      maxp = fmax(maxp, fabs(djj));
      minp = fmin(minp, fabs(djj));
      rank += 1;
    }
    a[6 * j + j] = 1.0;
  }
  for (int r = 0; r < 6; ++r)
    for (int c = r + 1; c < 6; ++c) a[6 * r + c] = 0.0;
  const double cond = rank == 0 ? 0.0 : minp / maxp;
  return (neg && cond < 1e-10) ? 2 : 0;
}

// The factor goes by panels of kFP = 48 columns (8 pose blocks), three launches
// each: the diagonal 48 x 48 block in one CTA, the rows below it (a thread
// each), the trailing triangle.  Every entry of S meets the 6-column steps in
// order, each as one difference with a sum over its six columns, so L and the
// pivots keep the bits of the step-by-step factor (two launches per step, 20 us
// for a step's 6 x 6 block in one thread).
//
// What shapes these kernels (measured on GB300): an SM sub-partition takes 64
// cycles for an FP64 instruction of a warp, however many of its lanes are
// active, and does not overlap two of them; a division is nine such, 566
// cycles.  So independent FP64 work goes to different lanes first (an entry a
// thread, the divisions of a row to six threads) and then to four warps.
constexpr int kFP = 48;

// ldlt6 by lanes 0 .. 5 of a warp, a row each (columns updated as soon as their
// pivot is known).  The rule compares a pivot with the largest pivot before the
// row in hand; the lanes compare it when it is formed, so a block in which a
// kept pivot is below that threshold of a later one is redone by lane 0 alone.
// a: 6x6 lower in shared memory (row stride ld); L6 (36), d6 (6) out.
__device__ __forceinline__ int ldlt6_warp(const double* a, int ld, double* L6, double* d6, int lane) {
  const unsigned all = 0xffffffffu;
  const int j = lane < 6 ? lane : 5;
  double v[6], l[6], d[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    v[c] = c <= j ? a[j * ld + c] : 0.0;
    l[c] = 0.0;
  }
  // magnitudes are compared by their bits (the same order): an FP64 comparison
  // takes the FP64 pipe's 70 cycles, and the pivots are a serial chain
  const long long kAbs = 0x7fffffffffffffffll, kInf = 0x7ff0000000000000ll;
  long long maxb = __double_as_longlong(1.0), minb = kInf;
  int rank = 0, st = 0;
  bool neg = false;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double tol = __longlong_as_double(maxb) * kCovTolRel;
    const double dk = __shfl_sync(all, v[k], k);
    const long long bits = __double_as_longlong(dk), ab = bits & kAbs;
    if (ab >= kInf && st == 0) st = 1;
    const double q = v[k] / dk;
    const bool zero = ab <= __double_as_longlong(tol);
    d[k] = zero ? 0.0 : dk;
    neg = neg || (!zero && bits < 0);
    maxb = zero ? maxb : max(maxb, ab);
    minb = zero ? minb : min(minb, ab);
    rank += zero ? 0 : 1;
    l[k] = zero ? 0.0 : q;
    const double ld_k = l[k] * d[k];
#pragma unroll
    for (int c = k + 1; c < 6; ++c) {
      const double lc = __shfl_sync(all, l[k], c);
      const double nv = v[c] - ld_k * lc;
      v[c] = c <= j ? nv : v[c];
    }
  }
  const double maxp = __longlong_as_double(maxb), minp = __longlong_as_double(minb);
  // minp <= tol of the largest pivot: a row may see an earlier pivot as zero
  if (st == 0 && rank > 0 && minp <= maxp * kCovTolRel) {
    if (lane == 0) {
      double b[36];
      for (int r = 0; r < 6; ++r)
        for (int c = 0; c < 6; ++c) b[6 * r + c] = c <= r ? a[r * ld + c] : 0.0;
      st = ldlt6(b, d);
      for (int e = 0; e < 36; ++e) L6[e] = b[e];
      for (int e = 0; e < 6; ++e) d6[e] = d[e];
    }
    __syncwarp();
    return __shfl_sync(all, st, 0);
  }
  if (lane < 6) {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      L6[6 * j + c] = c < j ? l[c] : (c == j ? 1.0 : 0.0);
      if (c == j) d6[j] = d[c];
    }
  }
  __syncwarp();
  if (st) return st;
  const double cond = rank == 0 ? 0.0 : minp / maxp;
  return (neg && cond < 1e-10) ? 2 : 0;
}

// y of a row's six columns from its entries x (L6 of the step): in place; L is
// y / d, formed by other threads (div6)
__device__ __forceinline__ void row_y6(double* x, const double* L6) {
  double yv[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    double v = x[j];
#pragma unroll
    for (int t = 0; t < j; ++t) v -= yv[t] * L6[6 * j + t];
    yv[j] = v;
  }
#pragma unroll
  for (int j = 1; j < 6; ++j) x[j] = yv[j];
}
__device__ __forceinline__ double div6(double y, double d) {
  const double q = y / d;
  return d == 0.0 ? 0.0 : q;
}

// The diagonal block of the panel at c0 (w columns): its 6-column steps in
// shared memory; L below the 6x6 blocks back to S.
__global__ void __launch_bounds__(kCovThreads) k_cov_diag(int n, int c0, int w, double* S, double* ldiag, double* dpiv,
                                                         int* status) {
  __shared__ double A[kFP][kFP + 1], Ld[kFP][7], L6[36], d6[6];
  const int tid = threadIdx.x;
  for (int e = tid; e < kFP * kFP; e += kCovThreads) {
    const int r = e / kFP, c = e % kFP;
    A[r][c] = (r < w && c <= r) ? S[static_cast<int64_t>(c0 + r) * n + c0 + c] : 0.0;
  }
  __syncthreads();
  for (int k0 = 0; k0 < w; k0 += 6) {
    if (tid < 32) {
      const int st = ldlt6_warp(&A[k0][k0], kFP + 1, L6, d6, tid);
      if (st && tid == 0) atomicMax(status, st);
      for (int e = tid; e < 36; e += 32) ldiag[6 * static_cast<int64_t>(c0 + k0) + e] = L6[e];
      if (tid < 6) dpiv[c0 + k0 + tid] = d6[tid];
    }
    __syncthreads();
    const int rows = w - k0 - 6;
    if (tid < rows) row_y6(&A[k0 + 6 + tid][k0], L6);
    __syncthreads();
    if (tid < 6 * rows) {
      const int r = tid / 6, t = tid - 6 * r;
      const double l = div6(A[k0 + 6 + r][k0 + t], d6[t]);
      A[k0 + 6 + r][k0 + t] = l;
      Ld[r][t] = l * d6[t];
    }
    __syncthreads();
    for (int e = tid; e < rows * (rows + 1) / 2; e += kCovThreads) {
      int i = static_cast<int>((sqrtf(8.0f * static_cast<float>(e) + 1.0f) - 1.0f) * 0.5f);
      while (i * (i + 1) / 2 > e) --i;
      while ((i + 1) * (i + 2) / 2 <= e) ++i;
      const double* li = &A[k0 + 6 + i][k0];
      const int j = e - i * (i + 1) / 2;
      double s = 0.0;
#pragma unroll
      for (int t = 0; t < 6; ++t) s += li[t] * Ld[j][t];
      A[k0 + 6 + i][k0 + 6 + j] -= s;
    }
    __syncthreads();
  }
  for (int e = tid; e < kFP * kFP; e += kCovThreads) {
    const int r = e / kFP, c = e % kFP;
    if (r < w && c / 6 < r / 6) S[static_cast<int64_t>(c0 + r) * n + c0 + c] = A[r][c];
  }
}

// The rows below the panel, 32 to a CTA: per step warp 0 forms y of every row
// (a thread each), the four warps share out the divisions, then the rows'
// entries in the panel's later columns.
constexpr int kRowsT = 128;
__global__ void __launch_bounds__(kRowsT) k_cov_rows(int n, int c0, double* S, const double* __restrict__ ldiag,
                                                    const double* __restrict__ dpiv) {
  extern __shared__ double sh[];
  double* Ld = sh;                      // kFP x kFP: L_jt d_t of the panel's own rows
  double* L6 = Ld + kFP * kFP;          // kFP / 6 x 36
  double* d = L6 + 6 * kFP;             // kFP
  double* X = d + kFP;                  // 32 x (kFP + 1)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r0 = c0 + kFP + blockIdx.x * 32;
  bool any = false;
#pragma unroll 12
  for (int e = tid; e < 32 * kFP; e += kRowsT) {
    const int r = e / kFP, c = e % kFP;
    const double v = r0 + r < n ? S[static_cast<int64_t>(r0 + r) * n + c0 + c] : 0.0;
    X[r * (kFP + 1) + c] = v;
    any = any || v != 0.0;
  }
  if (!__syncthreads_or(any)) return;  // rows outside the band: L is zero there
#pragma unroll 6
  for (int e = tid; e < kFP * kFP; e += kRowsT) {
    const int r = e / kFP, c = e % kFP;
    Ld[e] = c / 6 < r / 6 ? S[static_cast<int64_t>(c0 + r) * n + c0 + c] * dpiv[c0 + c] : 0.0;
  }
  for (int e = tid; e < kFP * 6; e += kRowsT) L6[e] = ldiag[6 * static_cast<int64_t>(c0) + e];
  if (tid < kFP) d[tid] = dpiv[c0 + tid];
  __syncthreads();
  double* x = X + lane * (kFP + 1);
  for (int k0 = 0; k0 < kFP; k0 += 6) {
    if (warp == 0) row_y6(x + k0, L6 + 6 * k0);
    __syncthreads();
    for (int t = warp; t < 6; t += 4) x[k0 + t] = div6(x[k0 + t], d[k0 + t]);
    __syncthreads();
    double l[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) l[t] = x[k0 + t];
    for (int j = k0 + 6 + 6 * warp; j < kFP; j += 24) {
      double s[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int u = 0; u < 6; ++u) s[u] += l[t] * Ld[(j + u) * kFP + k0 + t];
#pragma unroll
      for (int u = 0; u < 6; ++u) x[j + u] -= s[u];
    }
    __syncthreads();
  }
#pragma unroll 12
  for (int e = tid; e < 32 * kFP; e += kRowsT) {
    const int r = e / kFP, c = e % kFP;
    if (r0 + r < n) S[static_cast<int64_t>(r0 + r) * n + c0 + c] = X[r * (kFP + 1) + c];
  }
}
constexpr size_t kRowsSmem = sizeof(double) * (kFP * kFP + 6 * kFP + kFP + 32 * (kFP + 1));

// C_ij -= sum_t L_it (d_t L_jt), step by step of the panel, on the lower
// trailing triangle in 32 x 32 tiles (tiles above the diagonal, and tiles whose
// rows or columns are zero in the panel, return at once).
__global__ void __launch_bounds__(kCovThreads) k_cov_update(int n, int c0, double* S, const double* dpiv) {
  const int base = c0 + kFP;
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  __shared__ double Li[kUT][kFP + 1], Lj[kUT][kFP + 1];
  const int i0 = base + ti * kUT, j0 = base + tj * kUT;
  bool nzi = false, nzj = false;
  for (int e = threadIdx.x; e < kUT * kFP; e += blockDim.x) {
    const int r = e / kFP, t = e % kFP;
    const double vi = (i0 + r < n) ? S[static_cast<int64_t>(i0 + r) * n + c0 + t] : 0.0;
    const double vj = (j0 + r < n) ? S[static_cast<int64_t>(j0 + r) * n + c0 + t] : 0.0;
    nzi = nzi || vi != 0.0;
    nzj = nzj || vj != 0.0;
    Li[r][t] = vi;
    Lj[r][t] = vj * dpiv[c0 + t];
  }
  const int some = __syncthreads_or(nzi);
  if (!__syncthreads_or(nzj) || !some) return;
  const int jj = threadIdx.x & 31, i1 = threadIdx.x >> 5;
  const int j = j0 + jj;
  if (j >= n) return;
  double c[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = i0 + i1 + 8 * u;
    c[u] = (i < n && j <= i) ? S[static_cast<int64_t>(i) * n + j] : 0.0;
  }
  for (int k0 = 0; k0 < kFP; k0 += 6) {
    double s[4] = {0, 0, 0, 0};
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const double lj = Lj[jj][k0 + t];
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] += Li[i1 + 8 * u][k0 + t] * lj;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) c[u] -= s[u];
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = i0 + i1 + 8 * u;
    if (i < n && j <= i) S[static_cast<int64_t>(i) * n + j] = c[u];
  }
}

// ---------------------------------------------------------------------------
// Inverse from the factor: S^-1 = W^T D^-1 W with W = L^-1 (unit lower), in
// blocks of kIB = 48.  The diagonal blocks of W in one launch, then level by
// level (blocks of 1, 2, 4, .. kIB) W21 = -W22 (L21 W11) for all pairs of
// neighbouring blocks at once: two launches a level, then one for the product,
// in place of three for each of the n / 6 block rows of the Takahashi
// recurrence (28 ms of short, latency-bound launches at n = 1,788).  Tiles of
// L and of L21 W11 that are zero (outside the band of a loop) are skipped.
// The recurrence multiplies computed entries of the inverse, this does not:
// against 80-bit arithmetic its error is a tenth (1e-14 of the norm, 100 loop
// cameras).  W is kept transposed in the upper triangle of S; L21 W11 lives in
// Z until the product overwrites it.
// ---------------------------------------------------------------------------
constexpr int kIB = 48;
constexpr int kIBp = kIB + 1;
constexpr size_t kInvSmem = sizeof(double) * 3 * kIB * kIBp;

// W of the diagonal block b: inverses of its 6x6 blocks (a thread per column),
// then pairs of 6, 12, 24.  Rows past n: identity.  Also 1/d, and which tiles
// of block row b of L are not zero.
__global__ void __launch_bounds__(kCovThreads) k_cov_winv(int n, double* S, const double* __restrict__ ldiag,
                                                         const double* __restrict__ dpiv, double* __restrict__ dinv,
                                                         int* __restrict__ lnz, int nb) {
  extern __shared__ double sh[];
  double* L = sh;
  double* W = L + kIB * kIBp;
  double* T = W + kIB * kIBp;
  const int b = blockIdx.x, r0 = b * kIB, w = min(kIB, n - r0), tid = threadIdx.x;
  for (int e = tid; e < kIB * kIB; e += kCovThreads) {
    const int r = e / kIB, c = e % kIB;
    double v = r == c ? 1.0 : 0.0;
    if (r < w && c < r)
      v = r / 6 == c / 6 ? ldiag[36 * static_cast<int64_t>((r0 + r) / 6) + 6 * (r % 6) + c % 6]
                         : S[static_cast<int64_t>(r0 + r) * n + r0 + c];
    L[r * kIBp + c] = v;
    W[r * kIBp + c] = r == c ? 1.0 : 0.0;
  }
  if (tid < w) {
    const double d = dpiv[r0 + tid];
    dinv[r0 + tid] = d != 0.0 ? 1.0 / d : 0.0;
  }
  __syncthreads();
  if (tid < kIB) {
    const int c = tid, q0 = c / 6 * 6;
    for (int r = c + 1; r < q0 + 6; ++r) {
      double v = 0.0;
      for (int k = c; k < r; ++k) v -= L[r * kIBp + k] * W[k * kIBp + c];
      W[r * kIBp + c] = v;
    }
  }
  __syncthreads();
  for (int h = 6; h < kIB; h *= 2) {
    const int per = h * h, pairs = kIB / (2 * h);
    for (int e = tid; e < pairs * per; e += kCovThreads) {
      const int q = e / per, l0 = q * 2 * h, i = l0 + h + (e % per) / h, j = l0 + e % h;
      double v = 0.0;
      for (int k = j; k < l0 + h; ++k) v += L[i * kIBp + k] * W[k * kIBp + j];
      T[i * kIBp + j] = v;
    }
    __syncthreads();
    for (int e = tid; e < pairs * per; e += kCovThreads) {
      const int q = e / per, l0 = q * 2 * h, i = l0 + h + (e % per) / h, j = l0 + e % h;
      double v = 0.0;
      for (int k = l0 + h; k <= i; ++k) v -= W[i * kIBp + k] * T[k * kIBp + j];
      W[i * kIBp + j] = v;
    }
    __syncthreads();
  }
  for (int e = tid; e < kIB * kIB; e += kCovThreads) {
    const int c = e / kIB, r = e % kIB;
    if (c < r && r < w) S[static_cast<int64_t>(r0 + c) * n + r0 + r] = W[r * kIBp + c];
  }
  for (int K = 0; K < b; ++K) {
    bool any = false;
    for (int e = tid; e < kIB * kIB; e += kCovThreads) {
      const int r = e / kIB, c = e % kIB;
      if (r < w) any = any || S[static_cast<int64_t>(r0 + r) * n + K * kIB + c] != 0.0;
    }
    const int some = __syncthreads_or(any);
    if (tid == 0) lnz[b * nb + K] = some;
  }
}

// columns k0 .. k0 + nc - 1 of tile (I, K), I >= K, of W as dst[row][k - k0]:
// from the upper triangle of S
__device__ __forceinline__ void load_w(const double* S, int n, int I, int K, int k0, int nc, double* dst) {
#pragma unroll 6
  for (int e = threadIdx.x; e < kIB * nc; e += blockDim.x) {
    const int c = e / kIB, r = e % kIB;
    const int row = I * kIB + r, col = K * kIB + k0 + c;
    double v = 0.0;
    if (row < n && col < n) v = col < row ? S[static_cast<int64_t>(col) * n + row] : (col == row ? 1.0 : 0.0);
    dst[r * kIBp + c] = v;
  }
}

// Product of two tiles in shared memory, 3x3 entries a thread: rows ty + 16 i
// of A, columns tx + TX j of B (48 x 3 TX)
template <int TX>
__device__ __forceinline__ void tile_madd(const double* A, const double* B, double (*acc)[3]) {
  const int ty = threadIdx.x / TX, tx = threadIdx.x % TX;
#pragma unroll 4
  for (int k = 0; k < kIB; ++k) {
    double av[3], bv[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) av[i] = A[(ty + 16 * i) * kIBp + k];
#pragma unroll
    for (int j = 0; j < 3; ++j) bv[j] = B[k * kIBp + tx + TX * j];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[i][j] += av[i] * bv[j];
  }
}

// One level (left blocks of h tiles): M = 0: T = L21 W11 into Z, M = 1: W21 =
// -W22 T.  grid: x half a column tile of the left block, y the row tile of the
// right one, z the pair.  A tile product keeps an SM's FP64 pipe for 28 us, so
// a CTA takes 24 of the 48 columns (the dense rows of a loop closure are few
// long sums).
constexpr int kLvT = 128, kLvC = 24;
template <int M>
__global__ void __launch_bounds__(kLvT) k_cov_wlevel(int n, int nb, int h, double* S, double* Z,
                                                    const int* __restrict__ lnz, int* __restrict__ tnz) {
  extern __shared__ double sh[];
  __shared__ int s_nz[kLvT];
  double* A = sh;
  double* B = A + kIB * kIBp;
  const int left = blockIdx.z * 2 * h, I = left + h + blockIdx.y, J = left + (blockIdx.x >> 1);
  const int cc = (blockIdx.x & 1) * kLvC;
  if (I >= nb) return;
  const int tid = threadIdx.x;
  double acc[3][3] = {};
  bool any = false;
  const int k0 = M == 0 ? J : left + h, k1 = M == 0 ? left + h : I + 1;
  for (int K = k0; K < k1; ++K) {
    const int kk = (K - k0) % kLvT;
    if (kk == 0) {  // the next flags, all at once
      __syncthreads();
      if (K + tid < k1) s_nz[tid] = M == 0 ? lnz[I * nb + K + tid] : tnz[(K + tid) * nb + J];
      __syncthreads();
    }
    if (!s_nz[kk]) continue;  // uniform over the CTA
    any = true;
    __syncthreads();
    if (M == 0) {
#pragma unroll 6
      for (int e = tid; e < kIB * kIB; e += kLvT) {
        const int r = e / kIB, c = e % kIB, row = I * kIB + r;
        A[r * kIBp + c] = row < n ? S[static_cast<int64_t>(row) * n + K * kIB + c] : 0.0;
      }
      load_w(S, n, K, J, cc, kLvC, B);
    } else {
      load_w(S, n, I, K, 0, kIB, A);
#pragma unroll 3
      for (int e = tid; e < kIB * kLvC; e += kLvT) {
        const int r = e / kLvC, c = e % kLvC, row = K * kIB + r;
        B[r * kIBp + c] = row < n ? Z[static_cast<int64_t>(row) * n + J * kIB + cc + c] : 0.0;
      }
    }
    __syncthreads();
    tile_madd<8>(A, B, acc);
  }
  const int ty = tid >> 3, tx = tid & 7;
  if (M == 0) {
    if (tid == 0) tnz[I * nb + J] = any;  // the same from both halves
    if (!any) return;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int row = I * kIB + ty + 16 * i, col = J * kIB + cc + tx + 8 * j;
      if (row >= n) continue;
      if (M == 0) Z[static_cast<int64_t>(row) * n + col] = acc[i][j];
      else S[static_cast<int64_t>(col) * n + row] = any ? -acc[i][j] : 0.0;
    }
}

// Z_IJ = sum_{K >= I} W_KI^T D_K^-1 W_KJ, tiles I >= J, both triangles written.
// Tiles in order of I: the longest sums first.
__global__ void __launch_bounds__(kCovThreads) k_cov_wtw(int n, int nb, const double* __restrict__ S,
                                                        const double* __restrict__ dinv, double* __restrict__ Z) {
  extern __shared__ double sh[];
  double* A = sh;
  double* B = A + kIB * kIBp;
  const int q = blockIdx.x;
  int I = static_cast<int>((sqrtf(8.0f * static_cast<float>(q) + 1.0f) - 1.0f) * 0.5f);
  while (I * (I + 1) / 2 > q) --I;
  while ((I + 1) * (I + 2) / 2 <= q) ++I;
  const int J = q - I * (I + 1) / 2, tid = threadIdx.x;
  double acc[3][3] = {};
  for (int K = I; K < nb; ++K) {
    __syncthreads();
    for (int e = tid; e < kIB * kIB; e += kCovThreads) {
      const int r = e / kIB, c = e % kIB;
      const int m = K * kIB + c, ri = I * kIB + r, rj = J * kIB + r;  // W_m,ri and W_m,rj
      double vi = 0.0, vj = 0.0;
      if (m < n) {
        const double di = dinv[m];
        if (ri < n) vi = m > ri ? S[static_cast<int64_t>(ri) * n + m] : (m == ri ? 1.0 : 0.0);
        if (rj < n) vj = m > rj ? S[static_cast<int64_t>(rj) * n + m] * di : (m == rj ? di : 0.0);
      }
      A[r * kIBp + c] = vi;
      B[c * kIBp + r] = vj;
    }
    __syncthreads();
    tile_madd<16>(A, B, acc);
  }
  const int ty = tid >> 4, tx = tid & 15;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int row = I * kIB + ty + 16 * i, col = J * kIB + tx + 16 * j;
      if (row >= n || col > row) continue;
      Z[static_cast<int64_t>(row) * n + col] = acc[i][j];
      Z[static_cast<int64_t>(col) * n + row] = acc[i][j];
    }
}

// ---------------------------------------------------------------------------
// Pseudo-inverse pieces
// ---------------------------------------------------------------------------

// C[i][j] = sum_k A(i, k) w_k B(k, j) (w null: 1), A(i, k) = A[i a_i + k a_k],
// B(k, j) = B[k b_k + j b_j]; 64 x 64 tiles, 16 deep, 4 x 4 per thread.
__global__ void __launch_bounds__(256) k_cov_gemm(int M, int N, int K, const double* __restrict__ A, int64_t a_i,
                                                 int64_t a_k, const double* __restrict__ w,
                                                 const double* __restrict__ B, int64_t b_k, int64_t b_j,
                                                 double* __restrict__ C, int64_t ldc) {
  __shared__ double As[kGK][kGT + 1], Bs[kGK][kGT + 1];
  const int i0 = blockIdx.y * kGT, j0 = blockIdx.x * kGT;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double acc[4][4];
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
  for (int k0 = 0; k0 < K; k0 += kGK) {
    for (int e = threadIdx.x; e < kGK * kGT; e += blockDim.x) {
      const int kk = e / kGT, ii = e % kGT;
      const int k = k0 + kk;
      const int i = i0 + ii, j = j0 + ii;
      double v = (i < M && k < K) ? A[i * a_i + k * a_k] : 0.0;
      if (w && k < K) v *= w[k];
      As[kk][ii] = v;
      Bs[kk][ii] = (j < N && k < K) ? B[k * b_k + j * b_j] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < kGK; ++kk) {
      double av[4], bv[4];
      for (int r = 0; r < 4; ++r) av[r] = As[kk][ty + 16 * r];
      for (int c = 0; c < 4; ++c) bv[c] = Bs[kk][tx + 16 * c];
      for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) acc[r][c] += av[r] * bv[c];
    }
    __syncthreads();
  }
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * r, j = j0 + tx + 16 * c;
      if (i < M && j < N) C[i * ldc + j] = acc[r][c];
    }
}

// E (n x r): the columns J of the scalar unit-lower L (diagonal blocks from
// ldiag, the rest from the factored S).
__global__ void k_cov_build_e(int n, int r, const double* __restrict__ L, const double* __restrict__ ldiag,
                              const int32_t* __restrict__ J, double* __restrict__ E) {
  const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (e >= static_cast<int64_t>(n) * r) return;
  const int row = static_cast<int>(e / r), c = static_cast<int>(e % r);
  const int col = J[c];
  double v;
  if (row < col) v = 0.0;
  else if (row / 6 == col / 6) v = ldiag[36 * static_cast<int64_t>(row / 6) + 6 * (row % 6) + col % 6];
  else v = L[static_cast<int64_t>(row) * n + col];
  E[e] = v;
}

// rows / columns r..rp-1 of the padded G: identity
__global__ void k_cov_pad_identity(int r, int rp, double* G) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= rp * rp) return;
  const int i = e / rp, j = e % rp;
  if (i >= r || j >= r) G[e] = (i == j) ? 1.0 : 0.0;
}

__global__ void k_cov_recip(int r, const int32_t* __restrict__ J, const double* __restrict__ dpiv,
                            double* __restrict__ w) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < r) w[c] = 1.0 / dpiv[J[c]];
}

// ---------------------------------------------------------------------------
// Queries
// ---------------------------------------------------------------------------
struct CovQArgs {
  int nq, mode, nc, np, n;
  int nci, nk;  // free camera params: rows of their block in S (6) and their count (4 or 6); else 0, 0
  const int32_t* q;
  const int32_t* pose_fb;
  const int32_t* pt_mb;
  const int64_t* pt_g_begin;
  const int32_t* g_pose;
  const double* rec;
  const double* y;
  const double* vinv;
  const double* Z;
  const double* hdiag;
  const double* wc;   // free camera params: W_cq, Y_cq per marginalized point, H_cc, H_ca per free pose
  const double* yc;
  const double* hcc;
  const double* hcp;
  int n_eterm;
  const int32_t* eterm_fm;
  const int32_t* eterm_fn;
  const double* e_hmn;
  double* out;
  int32_t* dims;
};

// (kind, index) -> block: camera 0 (index 0, free params only) -> 0, pose 1
// -> free block, point 2 -> marg block; -1: none
__device__ __forceinline__ int cov_resolve(const CovQArgs& a, int kind, int idx, int* dim) {
  if (kind == 0 && idx == 0 && a.nci > 0) {
    *dim = a.nk;
    return 0;
  }
  if (kind == 1 && idx >= 0 && idx < a.nc) {
    *dim = 6;
    return a.pose_fb[idx];
  }
  if (kind == 2 && idx >= 0 && idx < a.np) {
    *dim = 3;
    return a.pt_mb[idx];
  }
  *dim = 0;
  return -1;
}

// Z row / column of a free variable's block: the camera at 0, pose fb after it
__device__ __forceinline__ int64_t cov_zoff(const CovQArgs& a, int kind, int blk) {
  return kind == 0 ? 0 : a.nci + 6 * static_cast<int64_t>(blk);
}

// t[c] = sum over the free blocks f of point pt (its terms with a free pose,
// shared out over the eight lanes of a group, then the camera when its params
// are free) of Z[row, f] Y_f[:, c]; every lane of the group gets the sums.
__device__ __forceinline__ void cov_row_times_y(const CovQArgs& a, int64_t row, int pt, int mb, int sub, double* t) {
  t[0] = t[1] = t[2] = 0.0;
  const double* zr = a.Z + row * a.n;
  for (int64_t g = a.pt_g_begin[pt] + sub; g < a.pt_g_begin[pt + 1]; g += 8) {
    const int gb = a.pose_fb[a.g_pose[g]];
    if (gb < 0) continue;
    const double* Y = a.y + 18 * g;
    const double* z = zr + a.nci + 6 * static_cast<int64_t>(gb);
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) t[c] += z[k] * Y[3 * k + c];
  }
  if (a.nci > 0 && sub == 0) {
    const double* Y = a.yc + 18 * static_cast<int64_t>(mb);
    for (int k = 0; k < a.nk; ++k)
      for (int c = 0; c < 3; ++c) t[c] += zr[k] * Y[3 * k + c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
    for (int off = 4; off > 0; off >>= 1) t[c] += __shfl_xor_sync(0xffffffffu, t[c], off);
}

// One CTA per query.  Blocks of points multiply rows of Z by the points' Y, a
// group of eight lanes per row: the rows are read together and the chain per
// lane is an eighth of a row (an entry per thread walked all of them: 0.82 ms
// for 128 points of 25 terms).
constexpr int kCovQT = 128;
__global__ void __launch_bounds__(kCovQT) k_cov_query(CovQArgs a) {
  const int qi = blockIdx.x;
  const int32_t* q = a.q + 4 * qi;
  int rd = 0, cd = 0;
  const int rb = cov_resolve(a, q[0], q[1], &rd), cb = cov_resolve(a, q[2], q[3], &cd);
  const int e = threadIdx.x;
  double* o = a.out + 36 * static_cast<int64_t>(qi);
  if (e < 36) o[e] = 0.0;
  __syncthreads();  // entries are written below by other threads
  if (rb < 0 || cb < 0) {
    if (e == 0) a.dims[2 * qi] = a.dims[2 * qi + 1] = 0;  // no block (the reference's None)
    return;
  }
  const int rk = q[0], ck = q[2];
  const bool rf = rk != 2, cf = ck != 2;  // free (camera or pose) or marginalized (point)
  const int64_t n = a.n;
  // a query on a point whose H_mm is singular has no covariance
  const bool bad = a.mode == 0 && ((!rf && isnan(a.vinv[9 * static_cast<int64_t>(rb)])) ||
                                   (!cf && isnan(a.vinv[9 * static_cast<int64_t>(cb)])));
  if (e == 0) {
    a.dims[2 * qi] = bad ? -1 : rd;
    a.dims[2 * qi + 1] = bad ? -1 : cd;
  }
  if (bad) return;
  const int rp = q[1], cp = q[3];  // the variables' own indices
  const int grp = e >> 3, sub = e & 7;
  if (a.mode == 0 && rf != cf) {
    // -(S^-1[free rows, :] H_fm) H_mm^-1 = -sum over the point's free blocks of Z[rows, block] Y
    const int fk = rf ? rk : ck, fbk = rf ? rb : cb, pt = rf ? cp : rp, mb = rf ? cb : rb, fd = rf ? rd : cd;
    const int pr = grp < fd ? grp : fd - 1;
    double t[3];
    cov_row_times_y(a, cov_zoff(a, fk, fbk) + pr, pt, mb, sub, t);
    if (grp < fd && sub < 3) {
      const double v = sub == 0 ? t[0] : (sub == 1 ? t[1] : t[2]);
      o[rf ? 3 * pr + sub : fd * sub + pr] = -v;
    }
    return;
  }
  if (a.mode == 0 && !rf && !cf) {
    // H_mm[i]^-1 delta_ij + sum over the free blocks g of point i and h of point j of Y_g^T Z[g, h] Y_h
    double v0 = 0.0, v8 = 0.0;  // entry sub, and entry 8 (lane 0 of the group)
    auto add = [&](const double* Yrow, const double* t) {
      v0 += Yrow[sub / 3] * (sub % 3 == 0 ? t[0] : (sub % 3 == 1 ? t[1] : t[2]));
      if (sub == 0) v8 += Yrow[2] * t[2];
    };
    const int64_t g0 = a.pt_g_begin[rp], nrow = 6 * (a.pt_g_begin[rp + 1] - g0);
    for (int64_t rr = grp; rr - grp < nrow; rr += kCovQT / 8) {  // uniform over the CTA: the sums use whole warps
      const int64_t g = g0 + (rr < nrow ? rr : 0) / 6;
      const int k = static_cast<int>((rr < nrow ? rr : 0) % 6);
      const int gb = a.pose_fb[a.g_pose[g]];
      double t[3];
      cov_row_times_y(a, gb < 0 ? 0 : a.nci + 6 * static_cast<int64_t>(gb) + k, cp, cb, sub, t);
      if (rr < nrow && gb >= 0) add(a.y + 18 * g + 3 * k, t);
    }
    if (a.nci > 0) {
      const int k = grp < a.nk ? grp : 0;
      double t[3];
      cov_row_times_y(a, k, cp, cb, sub, t);
      if (grp < a.nk) add(a.yc + 18 * static_cast<int64_t>(rb) + 3 * k, t);
    }
    __shared__ double part[kCovQT / 8][9];
    part[grp][sub] = v0;
    if (sub == 0) part[grp][8] = v8;
    __syncthreads();
    if (e < 9) {
      double v = 0.0;
      for (int w = 0; w < kCovQT / 8; ++w) v += part[w][e];
      if (rp == cp) v += a.vinv[9 * static_cast<int64_t>(rb) + e];
      o[e] = v;
    }
    return;
  }
  if (e >= rd * cd) return;
  const int r = e / cd, c = e % cd;
  double v = 0.0;
  if (a.mode == 1) {
    // precision: blocks of the undamped H
    if (rk == 0 && ck == 0) {
      v = a.hcc[6 * r + c];
    } else if (rk == 0 || ck == 0) {
      const int other = rk == 0 ? ck : rk, ob = rk == 0 ? cb : rb;
      const int cr = rk == 0 ? r : c, oc = rk == 0 ? c : r;  // camera row, the other block's column
      v = other == 1 ? a.hcp[36 * static_cast<int64_t>(ob) + 6 * cr + oc] : a.wc[18 * static_cast<int64_t>(ob) + 3 * cr + oc];
    } else if (rf && cf) {
      if (rb == cb) {
        v = a.hdiag[36 * static_cast<int64_t>(rb) + 6 * r + c];
      } else {
        for (int t = 0; t < a.n_eterm; ++t) {
          if (a.eterm_fm[t] == rb && a.eterm_fn[t] == cb) v += a.e_hmn[36 * static_cast<int64_t>(t) + 6 * r + c];
          if (a.eterm_fn[t] == rb && a.eterm_fm[t] == cb) v += a.e_hmn[36 * static_cast<int64_t>(t) + 6 * c + r];
        }
      }
    } else if (rf != cf) {
      const int pose = rf ? rp : cp, pt = rf ? cp : rp;
      const int pr = rf ? r : c, pc = rf ? c : r;  // (pose row, point column) of W
      for (int64_t g = a.pt_g_begin[pt]; g < a.pt_g_begin[pt + 1]; ++g)
        if (a.g_pose[g] == pose) v = a.rec[kCovRec * g + 21 + 3 * pr + pc];
    } else if (rp == cp) {
      for (int64_t g = a.pt_g_begin[rp]; g < a.pt_g_begin[rp + 1]; ++g)
        v += a.rec[kCovRec * g + 39 + (r <= c ? up_idx(3, r, c) : up_idx(3, c, r))];
    }
  } else {
    v = a.Z[(cov_zoff(a, rk, rb) + r) * n + cov_zoff(a, ck, cb) + c];
  }
  o[e] = v;
}

inline unsigned blocks_for(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

}  // namespace

int launch_cov_assemble(const Sizes& s, const Dev& d, const CovBufs& c, cudaStream_t st) {
  int nl = 0;
  if (s.ng > 0) {
    if (s.eucm)
      k_cov_groups<true><<<blocks_for(s.ng, kCovThreads), kCovThreads, 0, st>>>(s.ng, d.g_begin, d.g_pose, d.g_pt,
                                                                               d.poses, d.points, d.intr, c.rec,
                                                                               c.crec);
    else
      k_cov_groups<false><<<blocks_for(s.ng, kCovThreads), kCovThreads, 0, st>>>(s.ng, d.g_begin, d.g_pose, d.g_pt,
                                                                                d.poses, d.points, d.intr, c.rec,
                                                                                c.crec);
    ++nl;
  }
  if (s.np > 0) {
    k_cov_points<<<blocks_for(s.np, kCovPtT), kCovPtT, 0, st>>>(s.np, d.pt_g_begin, d.pt_mb, c.rec, c.vinv, c.status,
                                                               c.crec, c.wc, c.yc);
    ++nl;
    if (s.ng > 0) {
      k_cov_y<<<blocks_for(6 * s.ng, kCovThreads), kCovThreads, 0, st>>>(s.ng, d.g_pose, d.g_pt, d.pose_fb, d.pt_mb,
                                                                        c.rec, c.vinv, c.y);
      ++nl;
    }
  }
  if (c.crec) {
    k_cov_cam<<<1, kCovThreads, 0, st>>>(s.ng, s.nm, c.nk, c.n, c.crec, c.wc, c.yc, c.S, c.hcc);
    ++nl;
  }
  if (s.nsb > 0) {
    CovSArgs a{};
    a.nsb = s.nsb;
    a.n = c.n;
    a.sb_row = d.sb_row;
    a.sb_col = d.sb_col;
    a.fb_tile_begin = d.fb_tile_begin;
    a.tile_begin = d.tile_begin;
    a.tile_end = d.tile_end;
    a.cam_g = d.cam_g;
    a.cam_pt = c.cam_pt;
    a.pt_mb = d.pt_mb;
    a.rec = c.rec;
    a.y = c.y;
    a.prior_beg = s.n_prior > 0 ? d.prior_fb_begin : nullptr;
    a.prior_out = d.prior_out;
    a.e_beg = s.n_edge > 0 ? d.efb_begin : nullptr;
    a.e_slot = d.efb_slot;
    a.e_out = d.edge_out;
    a.eblk_begin = s.n_edge > 0 ? d.eblk_begin : nullptr;
    a.eblk_term = d.eblk_term;
    a.e_hmn = d.edge_hmn;
    a.S = c.S;
    a.hdiag = c.hdiag;
    a.nci = c.nci;
    a.crec = c.crec;
    a.wc = c.wc;
    a.hcp = c.hcp;
    if (c.ncam_g > 0) {
      k_cov_cam_pt<<<blocks_for(c.ncam_g, kCovThreads), kCovThreads, 0, st>>>(c.ncam_g, d.cam_g, d.g_pt, c.cam_pt);
      ++nl;
    }
    k_cov_s<<<static_cast<unsigned>(s.nsb), kCovSThreads, 0, st>>>(a);
    ++nl;
  }
  return nl;
}

int launch_cov_factor(int n, double* S, double* ldiag, double* dpiv, int* status, cudaStream_t st) {
  int nl = 0;
  for (int c0 = 0; c0 < n; c0 += kFP) {
    const int w = std::min(kFP, n - c0), below = n - c0 - w;
    k_cov_diag<<<1, kCovThreads, 0, st>>>(n, c0, w, S, ldiag, dpiv, status);
    ++nl;
    if (below > 0) {
      k_cov_rows<<<blocks_for(below, 32), kRowsT, kRowsSmem, st>>>(n, c0, S, ldiag, dpiv);
      const unsigned t = blocks_for(below, kUT);
      k_cov_update<<<dim3(t, t), kCovThreads, 0, st>>>(n, c0, S, dpiv);
      nl += 2;
    }
  }
  return nl;
}

// 1/d, then the nonzero-tile tables of L and of L21 W11
size_t cov_inverse_work(int n) {
  const size_t nb = static_cast<size_t>((n + kIB - 1) / kIB);
  return static_cast<size_t>(n) + nb * nb + 2;
}

cudaError_t launch_cov_inverse(int n, double* L, const double* ldiag, const double* dpiv, double* Z, double* work,
                               cudaStream_t st, int* launches) {
  const cudaError_t e = raise_dynamic_smem(reinterpret_cast<const void*>(k_cov_winv), kInvSmem);
  if (e != cudaSuccess) return e;
  const int nb = (n + kIB - 1) / kIB;
  double* dinv = work;
  int* lnz = reinterpret_cast<int*>(work + n);
  int* tnz = lnz + static_cast<size_t>(nb) * nb;
  constexpr size_t two = sizeof(double) * 2 * kIB * kIBp;
  k_cov_winv<<<nb, kCovThreads, kInvSmem, st>>>(n, L, ldiag, dpiv, dinv, lnz, nb);
  int nl = 1;
  for (int h = 1; h < nb; h *= 2) {
    const dim3 grid(2 * h, h, (nb + h - 1) / (2 * h));  // pairs whose right block exists
    k_cov_wlevel<0><<<grid, kLvT, two, st>>>(n, nb, h, L, Z, lnz, tnz);
    k_cov_wlevel<1><<<grid, kLvT, two, st>>>(n, nb, h, L, Z, lnz, tnz);
    nl += 2;
  }
  k_cov_wtw<<<nb * (nb + 1) / 2, kCovThreads, two, st>>>(n, nb, L, dinv, Z);
  if (launches) *launches += nl + 1;
  return cudaGetLastError();
}

namespace {
void gemm(int M, int N, int K, const double* A, int64_t a_i, int64_t a_k, const double* w, const double* B,
          int64_t b_k, int64_t b_j, double* C, int64_t ldc, cudaStream_t st) {
  if (M <= 0 || N <= 0) return;
  k_cov_gemm<<<dim3(blocks_for(N, kGT), blocks_for(M, kGT)), 256, 0, st>>>(M, N, K, A, a_i, a_k, w, B, b_k, b_j, C,
                                                                          ldc);
}
}  // namespace

cudaError_t cov_pinv(int n, const double* L, const double* ldiag, const double* dpiv, const std::vector<int32_t>& J,
                     double* Z, cudaMemPool_t pool, cudaStream_t st, int* g_ok) {
  *g_ok = 1;
  const int r = static_cast<int>(J.size());
  if (r == 0) return cudaMemsetAsync(Z, 0, sizeof(double) * n * static_cast<size_t>(n), st);
  const int rp = (r + 5) / 6 * 6;
  const size_t nr = static_cast<size_t>(n) * r;
  auto rnd = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t rr = static_cast<size_t>(r) * r, rpp = static_cast<size_t>(rp) * rp;
  const size_t bytes = rnd(sizeof(int32_t) * r) + 2 * rnd(sizeof(double) * nr) + 2 * rnd(sizeof(double) * rpp) +
                       rnd(sizeof(double) * rr) + rnd(sizeof(double) * r) + rnd(sizeof(double) * rp) +
                       rnd(sizeof(double) * (rp / 6) * 36) + rnd(sizeof(int) * 4) +
                       rnd(sizeof(double) * cov_inverse_work(rp));
  void* buf = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(&buf, bytes, pool, st);
  if (e != cudaSuccess) return e;
  char* p = static_cast<char*>(buf);
  auto take = [&p](size_t b) {
    void* v = p;
    p += (b + 255) / 256 * 256;
    return v;
  };
  int32_t* dJ = static_cast<int32_t*>(take(sizeof(int32_t) * r));
  double* E = static_cast<double*>(take(sizeof(double) * nr));
  double* F = static_cast<double*>(take(sizeof(double) * nr));
  double* G = static_cast<double*>(take(sizeof(double) * rp * rp));
  double* Gi = static_cast<double*>(take(sizeof(double) * rp * rp));
  double* M = static_cast<double*>(take(sizeof(double) * r * r));
  double* w = static_cast<double*>(take(sizeof(double) * r));
  double* gpiv = static_cast<double*>(take(sizeof(double) * rp));
  double* gdiag = static_cast<double*>(take(sizeof(double) * (rp / 6) * 36));
  int* gst = static_cast<int*>(take(sizeof(int) * 4));
  double* gwork = static_cast<double*>(take(sizeof(double) * cov_inverse_work(rp)));
  std::vector<double> hpiv(rp);
  e = cudaMemcpyAsync(dJ, J.data(), sizeof(int32_t) * r, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(gst, 0, sizeof(int) * 4, st);
  if (e == cudaSuccess) {
    k_cov_build_e<<<blocks_for(static_cast<int64_t>(nr), 256), 256, 0, st>>>(n, r, L, ldiag, dJ, E);
    // G = E^T E (r x r inside the rp x rp padded matrix, identity padding)
    gemm(r, r, n, E, 1, r, nullptr, E, r, 1, G, rp, st);
    k_cov_pad_identity<<<blocks_for(static_cast<int64_t>(rp) * rp, 256), 256, 0, st>>>(r, rp, G);
    launch_cov_factor(rp, G, gdiag, gpiv, gst, st);
    e = cudaMemcpyAsync(hpiv.data(), gpiv, sizeof(double) * rp, cudaMemcpyDeviceToHost, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) {
    for (int k = 0; k < r; ++k)
      if (!(hpiv[k] > 0.0)) *g_ok = 0;  // G is positive definite on the positive-pivot subspace
  }
  if (e == cudaSuccess && *g_ok) {
    e = launch_cov_inverse(rp, G, gdiag, gpiv, Gi, gwork, st, nullptr);
    k_cov_recip<<<blocks_for(r, 256), 256, 0, st>>>(r, dJ, dpiv, w);
    gemm(r, r, r, Gi, rp, 1, w, Gi, rp, 1, M, r, st);   // M = G^-1 diag(d_J)^-1 G^-1
    gemm(n, r, r, E, r, 1, nullptr, M, r, 1, F, r, st);  // F = E M
    gemm(n, n, r, F, r, 1, nullptr, E, 1, r, Z, n, st);  // Z = F E^T
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  const cudaError_t ef = cudaFreeAsync(buf, st);
  return e != cudaSuccess ? e : ef;
}

cudaError_t launch_cov_query(const Sizes& s, const Dev& d, const CovBufs& c, int mode, int nq, const int32_t* q,
                             double* out, int32_t* dims, cudaStream_t st) {
  if (nq <= 0) return cudaSuccess;
  CovQArgs a{};
  a.nq = nq;
  a.mode = mode;
  a.nc = s.nc;
  a.np = s.np;
  a.n = c.n;
  a.q = q;
  a.pose_fb = d.pose_fb;
  a.pt_mb = d.pt_mb;
  a.pt_g_begin = d.pt_g_begin;
  a.g_pose = d.g_pose;
  a.rec = c.rec;
  a.y = c.y;
  a.vinv = c.vinv;
  a.Z = c.Z;
  a.hdiag = c.hdiag;
  a.nci = c.nci;
  a.nk = c.nk;
  a.wc = c.wc;
  a.yc = c.yc;
  a.hcc = c.hcc;
  a.hcp = c.hcp;
  a.n_eterm = s.n_edge > 0 ? s.n_eterm : 0;
  a.eterm_fm = d.eterm_fm;
  a.eterm_fn = d.eterm_fn;
  a.e_hmn = d.edge_hmn;
  a.out = out;
  a.dims = dims;
  k_cov_query<<<nq, kCovQT, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace sgba
