// sgba_prior.cu -- cost functions on the poses alone, on the GPU: the pose
// prior (Isometry3PriorCostTerm,
// crates/sophus_opt/src/nlls/functor_library/costs/isometry3_prior.rs) and
// the pose-graph edge (PoseGraph3CostTerm, .../costs/pose_graph3.rs).
//
// Each prior k on pose j has a mean E_k and a 6x6 precision W_k; its residual
// is g = log(T_j E_k^-1) and its Jacobian J the derivative of
// log(exp(x) T_j E_k^-1) at x = 0, taken here in closed form, in
// f64 (sgba_lie.cuh: a direction per lane).  EvaluatedCostTerm::make
// (crates/sophus_opt/src/nlls/cost/evaluated_term.rs:286-327) then gives the
// Hessian block J^T W J, the gradient J^T W g and the cost g^T W g.  The
// priors are few (at most one group per pose) and run in f64; the
// blocks go to the pose's diagonal block in k_camera_finalize (damping once
// per pose with a prior: one reduced term of the prior cost function,
// cost_system.rs:229-236), the costs into extra partials of the merit and of
// the trial cost.
//
// Each edge on poses (m, n) with the measured pose_m_from_pose_n M has the
// residual g = log(T_m^-1 T_n M^-1), no precision and no robust kernel: cost
// g^T g.  With D the derivative of log(T_m^-1 exp(x) T_n M^-1) at x = 0
// (Isometry3::dx_log_a_exp_x_b_at_0), J_n = D and J_m = -D.  Edges with the
// same (m, n) form one reduced term: J_m^T J_m and J_n^T J_n (+ nu I once per
// term) go to the diagonal blocks, J_m^T J_n to the lower block of S between
// them (k_schur_reduce), -J^T g to the gradients (cost_system.rs:190-273).
#include <cuda_runtime.h>

#include <cstdint>

#include "sgba_dd.cuh"
#include "sgba_internal.h"
#include "sgba_lie.cuh"

namespace sgba {

namespace {

struct EdgeArgs {
  int nt;              // reduced terms
  const int32_t* tbeg; // nt + 1: edge ranges
  const int32_t* m;    // per edge
  const int32_t* n;
  const double* mn;    // per edge: pose_m_from_pose_n
  double* out;         // 2 nt records: J^T J (36), J^T g (6); side 0 pose m, side 1 pose n
  double* hmn;         // nt x 36: J_m^T J_n
};

__device__ __forceinline__ bool prior_halted(const Ctrl* c) { return c->done != 0; }
__device__ __forceinline__ bool prior_skipping(const Ctrl* c) { return c->done != 0 || c->skip != 0; }

// Eight lanes per term, one of the six tangent directions in each (two idle),
// and two warps per CTA, so that the terms lie on as many FP64 pipes as there
// are: a term's ~300 f64 operations, 64 cycles each whatever the lanes, bound
// the kernel.  (A thread per term with all six directions, in one CTA: 135 +
// 86 us an iteration of 151 poses, 150 edges and two priors; now 35 for both.)
constexpr int kTermLanes = 8;
constexpr int kTermThreads = 64;
constexpr int kTermsPerBlock = kTermThreads / kTermLanes;

__device__ __forceinline__ double term_shfl(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane, kTermLanes); }

__device__ __forceinline__ double pick3(const double* v, int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); }

// Residual g = log(q), its derivative d along this lane's direction k of x in
// A exp(x) B = (q, t), with A's rotation qa (identity: null) and B = b.
// `turned`: the signs of the product quaternion were turned.
__device__ __forceinline__ void term_log(const double* qa, const double* b, const double* ab, bool turned, int k,
                                         double* g, double* d) {
  // exp(x) B: the quaternion moves by (0, e_k / 2) b, the translation by e_k x t_b or e_k
  const int j = k % 3;
  double h[4] = {0.0, 0.0, 0.0, 0.0}, u[3], dq[4], dt[3];
  if (k < 3) {
    h[0] = -0.5 * pick3(b + 1, j);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int o = 3 - i - j;  // the third axis
      const bool next = i == j + 1 || (j == 2 && i == 0);  // e_j x v: -v_o at j + 1, +v_o at j + 2
      const double bq = pick3(b + 1, o), bt = pick3(b + 4, o);
      h[1 + i] = 0.5 * (i == j ? b[0] : (next ? -bq : bq));
      u[i] = i == j ? 0.0 : (next ? -bt : bt);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) u[i] = i == j ? 1.0 : 0.0;
  }
  if (qa) {
    lie::quat_mul(qa, h, dq);
    lie::rotate(qa, u, dt);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) dq[i] = h[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) dt[i] = u[i];
  }
  if (turned)
#pragma unroll
    for (int i = 0; i < 4; ++i) dq[i] = -dq[i];
  lie::se3_log(ab, dq, dt, g, d);
}

// CTAs [0, edge_blocks): reduced edge terms (the edges of a term in order); the
// others: priors (sorted by pose, constant poses last).  At `poses`; lin: the records of both sides
// and J_m^T J_n of a term, J^T W J and J^T W g of the priors on free poses
// (kPriorOut doubles each).  cost: a CTA's sum of g^T g and g^T W g in
// float-float to cost[blockIdx.x].  gate: 0 none, 1 the control block's done
// flag, 2 done or a skipped step.
__global__ void __launch_bounds__(kTermThreads) k_pose_terms(EdgeArgs ea, PriorArgs pa, int edge_blocks,
                                                             const double* __restrict__ poses, int lin, int gate,
                                                             double* cost, const Ctrl* ctrl) {
  if ((gate == 1 && prior_halted(ctrl)) || (gate == 2 && prior_skipping(ctrl))) return;
  const int k = threadIdx.x % kTermLanes, slot = threadIdx.x / kTermLanes;
  const int c = k < 6 ? k : 5;  // this lane's direction and column
  dd acc = dd_make(0.0f, 0.0f);
  if (static_cast<int>(blockIdx.x) < edge_blocks) {
    const int stride = edge_blocks * kTermsPerBlock;
    // whole warps loop together; a slot past the end repeats the last term and stores nothing
    for (int t0 = blockIdx.x * kTermsPerBlock; t0 < ea.nt; t0 += stride) {
      const bool on = t0 + slot < ea.nt;
      const int t = on ? t0 + slot : ea.nt - 1;
      double hcol[6], gc = 0.0;  // column c of D^T D, (D^T g)_c
#pragma unroll
      for (int i = 0; i < 6; ++i) hcol[i] = 0.0;
      const int e1 = ea.tbeg[t + 1];
      for (int e = ea.tbeg[t]; __any_sync(0xffffffffu, e < e1); ++e) {
        const bool live = e < e1;
        const int ei = live ? e : e1 - 1;
        double ai[7], mi[7], b[7], ab[7], g[6], d[6];
        lie::se3_inverse(poses + 7 * ea.m[ei], ai);
        lie::se3_inverse(ea.mn + 7 * ei, mi);
        lie::se3_mul(poses + 7 * ea.n[ei], mi, b);
        const bool turned = lie::se3_mul(ai, b, ab);
        term_log(ai, b, ab, turned, c, g, d);
        double cst = 0.0;
#pragma unroll
        for (int r = 0; r < 6; ++r) cst += g[r] * g[r];
        if (on && live && k == 0) acc = dd_add(acc, dd_from_double(cst));
        if (!lin) continue;
        // J_n = D, J_m = -D
        double sg = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) sg += d[q] * g[q];
        if (live) gc += sg;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
          double s2 = 0.0;
#pragma unroll
          for (int q = 0; q < 6; ++q) s2 += term_shfl(d[q], r) * d[q];
          if (live) hcol[r] += s2;
        }
      }
      if (lin && on && k < 6) {
        double* o0 = ea.out + static_cast<int64_t>(kPriorOut) * (2 * t);
        double* o1 = o0 + kPriorOut;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
          o0[6 * r + c] = hcol[r];
          o1[6 * r + c] = hcol[r];
          ea.hmn[36 * static_cast<int64_t>(t) + 6 * r + c] = -hcol[r];
        }
        o0[36 + c] = -gc;
        o1[36 + c] = gc;
      }
    }
  } else {
    const int stride = (gridDim.x - edge_blocks) * kTermsPerBlock;
    for (int p0 = (blockIdx.x - edge_blocks) * kTermsPerBlock; p0 < pa.n; p0 += stride) {
      const bool on = p0 + slot < pa.n;
      const int p = on ? p0 + slot : pa.n - 1;
      const double* W = pa.W + 36 * static_cast<int64_t>(p);
      double einv[7], te[7], g[6], d[6];
      lie::se3_inverse(pa.mean + 7 * p, einv);
      lie::se3_mul(poses + 7 * pa.pose[p], einv, te);
      term_log(nullptr, te, te, false, c, g, d);
      // lane r: (W g)_r
      double wr = 0.0;
#pragma unroll
      for (int q = 0; q < 6; ++q) wr += W[6 * c + q] * g[q];
      double wg[6];
#pragma unroll
      for (int r = 0; r < 6; ++r) wg[r] = term_shfl(wr, r);
      double cst = 0.0;
#pragma unroll
      for (int r = 0; r < 6; ++r) cst += g[r] * wg[r];
      if (on && k == 0) acc = dd_add(acc, dd_from_double(cst));
      if (!lin) continue;
      double wj[6], s = 0.0;  // column c of W J, (J^T W g)_c
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) v += W[6 * r + q] * d[q];
        wj[r] = v;
        s += d[r] * wg[r];
      }
      double* o = pa.out + static_cast<int64_t>(kPriorOut) * p;
      const bool store = on && k < 6 && pa.fb[p] >= 0;
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        double h = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) h += term_shfl(d[q], r) * wj[q];
        if (store) o[6 * r + c] = h;  // J^T W J
      }
      if (store) o[36 + c] = s;
    }
  }
  if (!cost) return;
  __shared__ float2 part[kTermThreads / 32];
  acc = dd_warp_sum(acc);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = make_float2(acc.hi, acc.lo);
  __syncthreads();
  if (threadIdx.x == 0)
    cost[blockIdx.x] = dd_to_double(dd_add(dd_make(part[0].x, part[0].y), dd_make(part[1].x, part[1].y)));
}

int term_blocks(int n) {
  const int b = (n + kTermsPerBlock - 1) / kTermsPerBlock;
  return b < kPoseTermMaxBlocks ? b : kPoseTermMaxBlocks;
}

// Equality constraints c_k = |t(T_k)| - r_k (TranslationNormConstraint,
// ba_scale_constraint.rs:57-100) at the current poses; under exp(x) T the
// translation moves by w x t + v, so the Jacobian is (0, t^T / |t|).  The
// KKT right-hand side gains G^T lambda on the free rows
// (eq_system.rs, populate_lower_triangular_kkt_mat): added here to the
// gradient and the reduced rhs in constraint order (one thread).
__global__ void k_eq_eval(int n, const int32_t* __restrict__ pose, const int32_t* __restrict__ fb,
                          const double* __restrict__ radius, const double* __restrict__ poses, double* c,
                          double* jac, const double* lambda, double* bf, double* rb, const Ctrl* ctrl) {
  if (prior_skipping(ctrl) || threadIdx.x != 0) return;
  for (int k = 0; k < n; ++k) {
    const double* t = poses + 7 * pose[k] + 4;
    const double nrm = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
    c[k] = nrm - radius[k];
    for (int i = 0; i < 3; ++i) jac[3 * k + i] = t[i] / nrm;
    if (fb[k] >= 0)
      for (int i = 0; i < 3; ++i) {
        bf[6 * fb[k] + 3 + i] += jac[3 * k + i] * lambda[k];
        rb[6 * fb[k] + 3 + i] += jac[3 * k + i] * lambda[k];
      }
  }
}

// The multiplier step's share of compute_gain_ratio's sums (its entries of
// the step against -c) and of the largest step entry.
__global__ void k_eq_post(int n, const double* __restrict__ dlam, const double* __restrict__ c, double* slot,
                          Ctrl* ctrl) {
  if (prior_skipping(ctrl) || threadIdx.x != 0) return;
  dd sdd = dd_make(0.f, 0.f), sdg = dd_make(0.f, 0.f);
  double mx = 0.0;
  for (int k = 0; k < n; ++k) {
    const dd x = dd_from_double(dlam[k]);
    sdd = dd_add(sdd, dd_mul(x, x));
    sdg = dd_add(sdg, dd_mul(x, dd_from_double(-c[k])));
    mx = fmax(mx, fabs(dlam[k]));
  }
  slot[0] = dd_to_double(sdd);
  slot[1] = dd_to_double(sdg);
  unsigned long long* addr = &ctrl->max_step_bits;
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(mx));
  atomicMax(addr, bits);  // non-negative doubles order as their bit patterns
}

}  // namespace

int launch_eq_eval(const Sizes& s, const Dev& d, cudaStream_t st) {
  if (s.n_eq <= 0) return 0;
  k_eq_eval<<<1, 32, 0, st>>>(s.n_eq, d.eq_pose, d.eq_fb, d.eq_radius, d.poses, d.eq_c, d.eq_jac, d.eq_lambda, d.bf,
                              d.rb, d.ctrl);
  return 1;
}

int launch_eq_post(const Sizes& s, const Dev& d, double* upd_slot, cudaStream_t st) {
  if (s.n_eq <= 0) return 0;
  k_eq_post<<<1, 32, 0, st>>>(s.n_eq, d.eq_dlam, d.eq_c, upd_slot, d.ctrl);
  return 1;
}

int pose_term_blocks(const Sizes& s) {
  return (s.n_edge > 0 ? term_blocks(s.n_eterm) : 0) + (s.n_prior > 0 ? term_blocks(s.n_prior) : 0);
}

int launch_pose_terms(const Sizes& s, const Dev& d, const double* poses, int lin, int gate, double* cost,
                      cudaStream_t st) {
  const int blocks = pose_term_blocks(s);
  if (blocks == 0) return 0;
  EdgeArgs ea{s.n_eterm, d.eterm_begin, d.edge_m, d.edge_n, d.edge_mn, d.edge_out, d.edge_hmn};
  PriorArgs pa{s.n_prior, d.prior_pose, d.prior_fb, d.prior_mean, d.prior_W, d.prior_out};
  k_pose_terms<<<blocks, kTermThreads, 0, st>>>(ea, pa, s.n_edge > 0 ? term_blocks(s.n_eterm) : 0, poses, lin, gate,
                                                cost, d.ctrl);
  return 1;
}

}  // namespace sgba
