// sgba_pcg.cu -- preconditioned conjugate gradients (PCG) on the reduced
// camera system S dx_f = b, with the exact LDL^T as the fallback.
//
// The reference solves the reduced system only exactly (block LDL^T,
// crates/sophus_solver/src/ldlt/schur_ldlt.rs:536-812, selected through the
// closed LinearSolverEnum, crates/sophus_solver/src/lib.rs:295-318).  This file
// adds an iterative alternative for the same step:
//   * Jacobi scaling S~ = D^-1/2 S D^-1/2 (D = diag S), b~ = D^-1/2 b;
//   * a block preconditioner per free pose: P_j = C_j^-T (I + L_j L_j^T) C_j^-1
//     with C_j the Cholesky factor of the 6x6 diagonal block of S~ (L_j = 0 is
//     block-Jacobi; L_j comes from the learned network, sgba_pcg_net.cu);
//   * CG with FP64 vectors and a float-float matrix-vector product, in one
//     cooperative launch (grid barriers with bounded waits; k_pcg_rows, or
//     k_pcg_solve for more or longer rows);
//     converged when |b~ - S~ x~| <= tol |b~|.  If it is not converged after
//     max_iters iterations (or breaks down, or a barrier wait gives up), the
//     exact factorization that follows in the same iteration runs as usual;
//     otherwise it is skipped (Ctrl::pcg_done).
// Every reduction uses a fixed partition and a fixed order: results are
// bit-reproducible.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "sgba_dd.cuh"
#include "sgba_internal.h"
#include "sgba_pcg_dev.cuh"

namespace sgba {

namespace {

constexpr int kPT = 512;                  // threads per CTA
constexpr int kPW = kPT / 32;             // warps per CTA
constexpr long long kBarSpins = 1ll << 22;  // x ~256 ns sleeps: a barrier wait gives up after ~1 s

__device__ __forceinline__ bool skipping(const Ctrl* c) { return c->done != 0 || c->skip != 0; }

// Float-float dot-product accumulator: the running sum through an exact
// TwoSum, the rounding errors of products and sums gathered in the lo part.
struct Acc {
  float hi, lo;
};
__device__ __forceinline__ void acc_madd(Acc& a, dd x, dd y) {
  const float pr = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -pr);
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  const float s = __fadd_rn(a.hi, pr);
  const float bb = __fsub_rn(s, a.hi);
  const float err = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(pr, bb));
  a.hi = s;
  a.lo = __fadd_rn(a.lo, __fadd_rn(err, e));
}
__device__ __forceinline__ dd acc_get(const Acc& a) { return dd_fast_two_sum(a.hi, a.lo); }

struct PcgArgs {
  int nf, n6;
  int64_t nsb;
  const int32_t* sb_row;
  const int32_t* sb_col;
  const int32_t* rowptr;
  const int32_t* cols;
  const int32_t* blks;
  const int32_t* diag;
  const double* S;     // dense n6 x n6 (both triangles of the pattern blocks)
  const double* rb;    // reduced right-hand side (unscaled)
  double* scl;
  double* Sb;
  float2* Sb2;         // the same blocks as float-float (hi, lo) pairs
  double* P;
  double* Cinv;
  const float* L;      // learned correction (nf * 21) or null
  double* vec;         // x r u p s w
  double* part;
  unsigned* bar;       // [0] arrivals (monotonic within a launch), [2] abort flag
  double* xout;
  float* xdd;
  int max_iters;
  double tol;
};

// ---------------------------------------------------------------- set-up ---

// The Jacobi scaling: a square root and a division per row (per entry of the
// blocks they took 17.6 us of 7,260 blocks; now 2.1 + 3.4).
__global__ void __launch_bounds__(128) k_pcg_scale(PcgArgs a, const Ctrl* ctrl) {
  if (skipping(ctrl)) return;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= a.n6) return;
  const double dr = a.S[static_cast<int64_t>(r) * a.n6 + r];
  a.scl[r] = (dr > 0.0 && isfinite(dr)) ? 1.0 / sqrt(dr) : 1.0;
}

// Jacobi-scaled lower blocks of S.
__global__ void __launch_bounds__(kPT) k_pcg_blocks(PcgArgs a, const Ctrl* ctrl) {
  if (skipping(ctrl)) return;
  const int64_t total = a.nsb * 36;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = t / 36;
    const int e = static_cast<int>(t % 36);
    const int r = 6 * a.sb_row[b] + e / 6, c = 6 * a.sb_col[b] + e % 6;
    const double v = a.S[static_cast<int64_t>(r) * a.n6 + c] * a.scl[r] * a.scl[c];
    a.Sb[t] = v;
    const dd vd = dd_from_double(v);
    a.Sb2[t] = make_float2(vd.hi, vd.lo);
  }
}

}  // namespace

namespace {

// pcg_precond_block by a warp, the same operations on each entry: lane i has
// row i of C, lane j column j of C^-1 (copies in lanes 8 g + j), and lanes
// 8 g + j form rows g and g + 4 of P's column j.  Bound by the serial square
// roots and divisions (35 us with a thread per pose, 11 so; 120 poses).
__global__ void __launch_bounds__(128) k_pcg_precond(PcgArgs a, const Ctrl* ctrl) {
  if (skipping(ctrl)) return;
  constexpr unsigned kAll = 0xffffffffu;
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (j >= a.nf) return;
  const int lane = threadIdx.x & 31, l = min(lane & 7, 5), g = lane >> 3;
  const bool own = (lane & 7) < 6;
  const double* B = a.Sb + 36 * static_cast<int64_t>(a.diag[j]);
  double* P = a.P + 36 * static_cast<int64_t>(j);
  double* Ci = a.Cinv + 36 * static_cast<int64_t>(j);
  double c[6], X[6];
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    double cq[6];  // row q of C
    double v = B[l * 6 + q];
#pragma unroll
    for (int k = 0; k < q; ++k) {
      cq[k] = __shfl_sync(kAll, c[k], q);
      v = fma(-c[k], cq[k], v);
    }
    const double d = __shfl_sync(kAll, v, q);
    if (!(d > 0.0) || !isfinite(d)) ok = false;  // the whole warp
    const double cqq = sqrt(d);
    c[q] = l < q ? 0.0 : (l == q ? cqq : v / cqq);
  }
  if (!ok) {
    if (g == 0 && own)
      for (int i = 0; i < 6; ++i) P[i * 6 + l] = Ci[i * 6 + l] = i == l ? 1.0 : 0.0;
    return;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < i; ++k) v = fma(-__shfl_sync(kAll, c[k], i), X[k], v);  // X[k] = 0 above the diagonal
    const double q = (i == l ? 1.0 : v) / __shfl_sync(kAll, c[i], i);
    X[i] = i < l ? 0.0 : q;
  }
  double T[6];
  if (a.L) {
    // M = I + L L^T, L lower 6x6 packed row-wise: column l of M, then T = M C^-1
    const float* L = a.L + kPcgOut * static_cast<int64_t>(j);
    double M[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double li = k <= i ? static_cast<double>(L[i * (i + 1) / 2 + k]) : 0.0;
        const double lj = k <= l ? static_cast<double>(L[l * (l + 1) / 2 + k]) : 0.0;
        v = fma(li, lj, v);
      }
      M[i] = (i == l ? 1.0 : 0.0) + v;
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) v = fma(__shfl_sync(kAll, M[i], k), X[k], v);
      T[i] = v;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) T[i] = X[i];
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = g + 4 * h;
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) v = fma(__shfl_sync(kAll, X[k], i < 6 ? i : 5), T[k], v);
    if (own && i < 6) P[i * 6 + l] = v;
  }
  if (g == 0 && own)
#pragma unroll
    for (int i = 0; i < 6; ++i) Ci[i * 6 + l] = X[i];
}

// ------------------------------------------------------------------ solve ---

// Grid barrier for a cooperative launch: a monotonic arrival counter; the
// k-th barrier of a launch waits until k * gridDim CTAs have arrived (the
// counter is zeroed before the launch).  Every wait is bounded: after
// kBarSpins polls the CTA sets the abort flag and returns false; every CTA
// also returns false once it sees the flag.
__device__ bool grid_barrier(unsigned* bar, unsigned target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    int ok = 1;
    long long spins = 0;
    unsigned v;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v >= target) break;
      unsigned ab;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(ab) : "l"(bar + 2) : "memory");
      if (ab != 0u) { ok = 0; break; }
      if (++spins > kBarSpins) {
        atomicExch(bar + 2, 1u);
        ok = 0;
        break;
      }
      if (spins > 64) __nanosleep(64);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Sum of one partial per CTA (slot k of kSlots), the same fixed order in
// every CTA.
constexpr int kSlots = 4;
__device__ void sum_parts3(const double* part, double* out) {
  __shared__ double s_sum[3];
  if (threadIdx.x < 32) {
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
    for (int g = threadIdx.x; g < static_cast<int>(gridDim.x); g += 32) {
      v0 += __ldcg(part + kSlots * g + 0);
      v1 += __ldcg(part + kSlots * g + 1);
      v2 += __ldcg(part + kSlots * g + 2);
    }
    for (int off = 16; off > 0; off >>= 1) {
      v0 += __shfl_down_sync(0xffffffffu, v0, off);
      v1 += __shfl_down_sync(0xffffffffu, v1, off);
      v2 += __shfl_down_sync(0xffffffffu, v2, off);
    }
    if (threadIdx.x == 0) {
      s_sum[0] = v0;
      s_sum[1] = v1;
      s_sum[2] = v2;
    }
  }
  __syncthreads();
  out[0] = s_sum[0];
  out[1] = s_sum[1];
  out[2] = s_sum[2];
  __syncthreads();
}

// Per-CTA partials of three dot products: warp sums combined in warp order.
__device__ void write_parts3(double* part, double v0, double v1, double v2) {
  __shared__ double s[3][kPW];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int off = 16; off > 0; off >>= 1) {
    v0 += __shfl_down_sync(0xffffffffu, v0, off);
    v1 += __shfl_down_sync(0xffffffffu, v1, off);
    v2 += __shfl_down_sync(0xffffffffu, v2, off);
  }
  if (lane == 0) {
    s[0][w] = v0;
    s[1][w] = v1;
    s[2][w] = v2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int q = 0; q < kPW; ++q) t += s[threadIdx.x][q];
    part[kSlots * blockIdx.x + threadIdx.x] = t;
  }
}

// w_j = sum over the full block row j of S~_jk u_k in float-float (the blocks
// as (hi, lo) FP32 pairs: FP64 runs at 1/64 of the FP32 rate here): lanes
// take entries, each lane forms the six rows of its block product, then a
// fixed shuffle tree.  Returns the six sums in every lane.
__device__ __forceinline__ void block_row_matvec(const PcgArgs& a, int j, const double* u, double* w6) {
  const int lane = threadIdx.x & 31;
  Acc acc[6];
#pragma unroll
  for (int r = 0; r < 6; ++r) acc[r] = Acc{0.0f, 0.0f};
  for (int e = a.rowptr[j] + lane; e < a.rowptr[j + 1]; e += 32) {
    const int k = a.cols[e];
    const int bi = a.blks[e];
    const bool tr = bi < 0;
    const float4* B4 = reinterpret_cast<const float4*>(a.Sb2 + 36 * static_cast<int64_t>(bi & 0x7fffffff));
    dd uk[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) uk[c] = dd_from_double(__ldcg(u + 6 * k + c));
#pragma unroll
    for (int h = 0; h < 18; ++h) {
      const float4 v = B4[h];  // entries 2h, 2h + 1 as (hi, lo)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = 2 * h + q;
        const int rr = tr ? t % 6 : t / 6, cc = tr ? t / 6 : t % 6;
        acc_madd(acc[rr], q ? dd_make(v.z, v.w) : dd_make(v.x, v.y), uk[cc]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    dd t = acc_get(acc[r]);
    for (int off = 16; off > 0; off >>= 1)
      t = dd_add(t, dd_make(__shfl_xor_sync(0xffffffffu, t.hi, off), __shfl_xor_sync(0xffffffffu, t.lo, off)));
    w6[r] = dd_to_double(t);
  }
}

// z = P_j r_j for the row's six entries (lane < 6 holds r_{6j+lane}).
__device__ __forceinline__ double precond_row(const PcgArgs& a, int j, double rv) {
  const int lane = threadIdx.x & 31;
  double zv = 0.0;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const double rc = __shfl_sync(0xffffffffu, rv, c);
    if (lane < 6) zv = fma(a.P[36 * static_cast<int64_t>(j) + lane * 6 + c], rc, zv);
  }
  return zv;
}

__device__ void pcg_report(Ctrl* ctrl, bool conv, bool ok, int it, int status, double bnorm2, double rr) {
  ctrl->pcg_done = conv ? 1 : 0;
  ctrl->pcg_iters = it;
  ctrl->pcg_status = status;
  ctrl->pcg_relres = (bnorm2 > 0.0 && ok) ? sqrt(rr / bnorm2) : 0.0;
  ctrl->pcg_solves += 1;
  ctrl->pcg_fallbacks += conv ? 0 : 1;
  ctrl->pcg_total_iters += it;
}

// PCG in the single-reduction form of Chronopoulos and Gear ("s-step
// iterative methods for symmetric linear systems", 1989): one matrix-vector
// product and one fused reduction of (r, u), (w, u), (r, r) per iteration,
// two grid barriers.  x~ solves S~ x~ = b~ (Jacobi-scaled).
__global__ void __launch_bounds__(kPT) k_pcg_solve(PcgArgs a, Ctrl* ctrl) {
  if (skipping(ctrl)) return;
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * kPW + (threadIdx.x >> 5);
  const int nw = gridDim.x * kPW;
  const unsigned nb = gridDim.x;
  unsigned nbar = 0;
  double* x = a.vec;
  double* r = a.vec + a.n6;
  double* u = a.vec + 2 * a.n6;
  double* p = a.vec + 3 * a.n6;
  double* sv = a.vec + 4 * a.n6;  // s = S~ p
  double* w = a.vec + 5 * a.n6;   // w = S~ u
  // x = 0, r = b~, u = P r
  for (int j = gw; j < a.nf; j += nw) {
    double rv = 0.0;
    if (lane < 6) {
      const int i = 6 * j + lane;
      rv = (a.scl ? a.scl[i] : 1.0) * a.rb[i];
      x[i] = 0.0;
      r[i] = rv;
      p[i] = 0.0;
      sv[i] = 0.0;
    }
    const double zv = precond_row(a, j, rv);
    if (lane < 6) u[6 * j + lane] = zv;
  }
  bool ok = grid_barrier(a.bar, (++nbar) * nb);
  double gamma = 0.0, alpha = 0.0, bnorm2 = 0.0, rr = 0.0;
  int it = 0;
  int status = ok ? 1 : 3;
  for (;;) {
    if (!ok) { status = 3; break; }
    // w = S~ u; dots (r, u), (w, u), (r, r)
    double ru = 0.0, wu = 0.0, r2 = 0.0;
    for (int j = gw; j < a.nf; j += nw) {
      double w6[6];
      block_row_matvec(a, j, u, w6);
      if (lane < 6) {
        const int i = 6 * j + lane;
        const double wv = w6[lane], uv = u[i], rv = r[i];
        w[i] = wv;
        ru += rv * uv;
        wu += wv * uv;
        r2 += rv * rv;
      }
    }
    write_parts3(a.part, ru, wu, r2);
    if (!(ok = grid_barrier(a.bar, (++nbar) * nb))) { status = 3; break; }
    double sums[3];
    sum_parts3(a.part, sums);
    const double gamma_n = sums[0], delta = sums[1];
    rr = sums[2];
    if (it == 0) bnorm2 = rr;
    if (!(bnorm2 > 0.0)) { status = 0; break; }  // b = 0: x = 0 is exact
    if (rr <= a.tol * a.tol * bnorm2) { status = 0; break; }
    if (it >= a.max_iters) { status = 1; break; }
    double beta;
    if (it == 0) {
      beta = 0.0;
      alpha = gamma_n / delta;
    } else {
      beta = gamma_n / gamma;
      alpha = gamma_n / (delta - beta * gamma_n / alpha);
    }
    gamma = gamma_n;
    if (!(alpha > 0.0) || !isfinite(alpha) || !(gamma_n > 0.0)) { status = 2; break; }
    // p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = P r
    for (int j = gw; j < a.nf; j += nw) {
      double rv = 0.0;
      if (lane < 6) {
        const int i = 6 * j + lane;
        const double pv = fma(beta, p[i], u[i]);
        const double sn = fma(beta, sv[i], w[i]);
        p[i] = pv;
        sv[i] = sn;
        x[i] = fma(alpha, pv, x[i]);
        rv = fma(-alpha, sn, r[i]);
        r[i] = rv;
      }
      const double zv = precond_row(a, j, rv);
      if (lane < 6) u[6 * j + lane] = zv;
    }
    ++it;
    if (!(ok = grid_barrier(a.bar, (++nbar) * nb))) { status = 3; break; }
  }
  const bool conv = ok && status == 0;
  if (conv) {
    for (int j = gw; j < a.nf; j += nw) {
      if (lane < 6) {
        const int i = 6 * j + lane;
        const double v = (a.scl ? a.scl[i] : 1.0) * x[i];
        if (a.xout) a.xout[i] = v;
        if (a.xdd) {
          const dd vd = dd_from_double(v);
          a.xdd[2 * i] = vd.hi;
          a.xdd[2 * i + 1] = vd.lo;
        }
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && ctrl) pcg_report(ctrl, conv, ok, it, status, bnorm2, rr);
}

// The same for up to 32 CTAs' worth of rows (k_pcg_solve's CTAs of 16 rows) and
// rows whose blocks fit in shared memory: four warps a CTA, a row per warp, so
// that the FP64 work of the vectors (64 cycles a warp instruction) and the
// products lie on four times the SMs.  A row's blocks stay in shared memory for
// the whole solve, transposed where the row needs the transpose, a block's pairs
// strided so that lanes read contiguous 16-byte words; x, r, p, s and the row of
// P stay in registers; u is exchanged as float-float pairs.  Sums are formed in
// k_pcg_solve's order (per 16 rows, then over those groups): the same bits.
// 120 poses, dense S: 812 -> 222 us a solve.
constexpr int kRowWarps = 4;
constexpr int kRowGroups = 32;  // groups of kPW rows at most
constexpr int kRowMax = kPW * kRowGroups;
static_assert(3 * kRowMax <= kSlots * kPcgMaxGrid, "the rows' partials fit");

__host__ __device__ constexpr size_t rows_smem(int nf, int row_max) {
  return 16 * (3 * static_cast<size_t>(nf) + 18 * static_cast<size_t>(kRowWarps) * row_max);
}

__global__ void __launch_bounds__(32 * kRowWarps, 1) k_pcg_rows(PcgArgs a, int row_max, Ctrl* ctrl) {
  if (skipping(ctrl)) return;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ float4 rows_sm[];
  __shared__ double s_sum[3];
  float2* us = reinterpret_cast<float2*>(rows_sm);  // u, 6 pairs a pose
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float4* B = rows_sm + 3 * a.nf + 18 * static_cast<size_t>(row_max) * w;
  const int j = blockIdx.x * kRowWarps + w;
  const bool on = j < a.nf;
  const unsigned nb = gridDim.x;
  const int groups = gridDim.x / (kPW / kRowWarps);
  unsigned nbar = 0;
  float2* u = reinterpret_cast<float2*>(a.vec + 2 * a.n6);
  const int e0 = on ? a.rowptr[j] : 0, len = on ? a.rowptr[j + 1] - e0 : 0;
  for (int i = lane; i < len; i += 32) {
    const int bi = a.blks[e0 + i];
    const float4* b4 = reinterpret_cast<const float4*>(a.Sb2 + 36 * static_cast<int64_t>(bi & 0x7fffffff));
    float2 v[36];
#pragma unroll
    for (int h = 0; h < 18; ++h) {
      const float4 t = b4[h];
      v[2 * h] = make_float2(t.x, t.y);
      v[2 * h + 1] = make_float2(t.z, t.w);
    }
#pragma unroll
    for (int h = 0; h < 18; ++h) {
      const int r = 2 * h / 6, c = 2 * h % 6;
      const float2 p = bi < 0 ? v[6 * c + r] : v[2 * h], q = bi < 0 ? v[6 * c + 6 + r] : v[2 * h + 1];
      B[h * len + i] = make_float4(p.x, p.y, q.x, q.y);
    }
  }
  // lane c < 6: entry 6 j + c of the vectors, row c of P_j
  const bool ent = on && lane < 6;
  const int64_t row = 6 * static_cast<int64_t>(j) + lane;
  double Pr[6], x = 0.0, r = 0.0, p = 0.0, sv = 0.0, uv = 0.0;
#pragma unroll
  for (int c = 0; c < 6; ++c) Pr[c] = ent ? a.P[36 * static_cast<int64_t>(j) + lane * 6 + c] : 0.0;
  auto precond = [&]() {  // u = P r
    uv = 0.0;
#pragma unroll
    for (int c = 0; c < 6; ++c) uv = fma(Pr[c], __shfl_sync(kAll, r, c), uv);
    if (ent) {
      const dd t = dd_from_double(uv);
      __stcg(u + row, make_float2(t.hi, t.lo));
    }
  };
  if (ent) r = (a.scl ? a.scl[row] : 1.0) * a.rb[row];
  precond();
  bool ok = grid_barrier(a.bar, (++nbar) * nb);
  double gamma = 0.0, alpha = 0.0, bnorm2 = 0.0, rr = 0.0;
  int it = 0;
  int status = ok ? 1 : 3;
  for (;;) {
    if (!ok) { status = 3; break; }
    for (int i = threadIdx.x; i < 3 * a.nf; i += 32 * kRowWarps)
      rows_sm[i] = __ldcg(reinterpret_cast<const float4*>(u) + i);
    __syncthreads();
    // w = S~ u
    Acc acc[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = Acc{0.0f, 0.0f};
    for (int i = lane; i < len; i += 32) {
      const float2* uk = us + 6 * a.cols[e0 + i];
      dd ud[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) ud[c] = dd_make(uk[c].x, uk[c].y);
#pragma unroll
      for (int h = 0; h < 18; ++h) {
        const float4 v = B[h * len + i];
        acc_madd(acc[2 * h / 6], dd_make(v.x, v.y), ud[2 * h % 6]);
        acc_madd(acc[2 * h / 6], dd_make(v.z, v.w), ud[2 * h % 6 + 1]);
      }
    }
    // the tree over the lanes (xor 16, 8, 4, 2, 1) with the six sums dealt out on
    // the way: sum q ends in the lanes 16 (q / 3) + 8 ((q % 3) / 2) + 4 ((q % 3) % 2) + 0 .. 3
    dd t[4];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
    auto swap = [&](dd keep, dd send, int off) {
      return dd_add(keep, dd_make(__shfl_xor_sync(kAll, send.hi, off), __shfl_xor_sync(kAll, send.lo, off)));
    };
    auto pick = [](bool b, dd y, dd n) { return dd_make(b ? y.hi : n.hi, b ? y.lo : n.lo); };
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const dd lo = acc_get(acc[q]), hi = acc_get(acc[3 + q]);
      t[q] = swap(pick(h16, hi, lo), pick(h16, lo, hi), 16);
    }
    t[3] = dd_make(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 2; ++q) t[q] = swap(pick(h8, t[2 + q], t[q]), pick(h8, t[q], t[2 + q]), 8);
    t[0] = swap(pick(h4, t[1], t[0]), pick(h4, t[0], t[1]), 4);
    t[0] = swap(t[0], t[0], 2);
    t[0] = swap(t[0], t[0], 1);
    const double ws = dd_to_double(t[0]);
    const int m = lane % 3, src = lane < 6 ? 16 * (lane / 3) + 8 * (m / 2) + 4 * (m % 2) : 0;
    const double wv = __shfl_sync(kAll, ws, src);  // lane c < 6: w_{6 j + c}
    // (r, u), (w, u), (r, r) in lanes 0, 8, 16
    {
      const int c = lane & 7;
      const double ra = __shfl_sync(kAll, r, c), ua = __shfl_sync(kAll, uv, c), wa = __shfl_sync(kAll, wv, c);
      double v = (on && c < 6) ? ((lane & 8) ? wa : ra) * ((lane & 16) ? ra : ua) : 0.0;
      v += __shfl_down_sync(kAll, v, 4, 8);
      v += __shfl_down_sync(kAll, v, 2, 8);
      v += __shfl_down_sync(kAll, v, 1, 8);
      if (c == 0 && lane < 24) __stcg(a.part + (lane >> 3) * kRowMax + j, v);
    }
    if (!(ok = grid_barrier(a.bar, (++nbar) * nb))) { status = 3; break; }
    if (w < 3) {
      double v = 0.0;
      if (lane < groups) {
        const double2* pp = reinterpret_cast<const double2*>(a.part + w * kRowMax + kPW * lane);
        double2 q[kPW / 2];
#pragma unroll
        for (int k = 0; k < kPW / 2; ++k) q[k] = __ldcg(pp + k);
#pragma unroll
        for (int k = 0; k < kPW / 2; ++k) {
          v += q[k].x;
          v += q[k].y;
        }
      }
      for (int off = 16; off > 0; off >>= 1)
        if (off < groups) v += __shfl_down_sync(kAll, v, off);
      if (lane == 0) s_sum[w] = v;
    }
    __syncthreads();
    const double gamma_n = s_sum[0], delta = s_sum[1];
    rr = s_sum[2];
    if (it == 0) bnorm2 = rr;
    if (!(bnorm2 > 0.0)) { status = 0; break; }  // b = 0: x = 0 is exact
    if (rr <= a.tol * a.tol * bnorm2) { status = 0; break; }
    if (it >= a.max_iters) { status = 1; break; }
    double beta;
    if (it == 0) {
      beta = 0.0;
      alpha = gamma_n / delta;
    } else {
      beta = gamma_n / gamma;
      alpha = gamma_n / (delta - beta * gamma_n / alpha);
    }
    gamma = gamma_n;
    if (!(alpha > 0.0) || !isfinite(alpha) || !(gamma_n > 0.0)) { status = 2; break; }
    // p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = P r
    p = fma(beta, p, uv);
    sv = fma(beta, sv, wv);
    x = fma(alpha, p, x);
    r = fma(-alpha, sv, r);
    precond();
    ++it;
    if (!(ok = grid_barrier(a.bar, (++nbar) * nb))) { status = 3; break; }
  }
  const bool conv = ok && status == 0;
  if (conv && ent) {
    const double v = (a.scl ? a.scl[row] : 1.0) * x;
    if (a.xout) a.xout[row] = v;
    if (a.xdd) {
      const dd vd = dd_from_double(v);
      a.xdd[2 * row] = vd.hi;
      a.xdd[2 * row + 1] = vd.lo;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && ctrl) pcg_report(ctrl, conv, ok, it, status, bnorm2, rr);
}

PcgArgs pcg_args(const Sizes& s, const Dev& d) {
  PcgArgs a;
  a.nf = s.nf;
  a.n6 = s.n6;
  a.nsb = s.nsb;
  a.sb_row = d.sb_row;
  a.sb_col = d.sb_col;
  a.rowptr = d.pcg_rowptr;
  a.cols = d.pcg_cols;
  a.blks = d.pcg_blks;
  a.diag = d.pcg_diag;
  a.S = d.S;
  a.rb = d.rb;
  a.scl = d.pcg_scl;
  a.Sb = d.pcg_S;
  a.Sb2 = d.pcg_S2;
  a.P = d.pcg_P;
  a.Cinv = d.pcg_Cinv;
  a.L = (s.pcg_mode == 2) ? d.pcg_L : nullptr;
  a.vec = d.pcg_vec;
  a.part = d.pcg_part;
  a.bar = d.pcg_bar;
  a.xout = d.x;
  a.xdd = d.xdd;
  a.max_iters = s.pcg_max_iters;
  a.tol = s.pcg_tol;
  return a;
}

}  // namespace

int pcg_setup(int nf, int* grid) {
  int dev = 0, sms = 0, per_sm = 0, coop = 0;
  *grid = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return -1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pcg_solve, kPT, 0) != cudaSuccess || per_sm < 1)
    return -1;
  const int want = (nf + kPW - 1) / kPW;
  int cap = sms * (per_sm < 2 ? per_sm : 2);
  if (cap > kPcgMaxGrid) cap = kPcgMaxGrid;
  *grid = want < cap ? (want > 0 ? want : 1) : cap;
  return 0;
}

// k_pcg_rows takes the system: its rows fit (one wave of CTAs, one per SM at most).
bool pcg_rows_setup(int nf, int row_max) {
  const size_t bytes = rows_smem(nf, row_max);
  if (nf > kRowMax || row_max < 1 || bytes > 220 * 1024) return false;
  if (cudaFuncSetAttribute(k_pcg_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  return (nf + kPW - 1) / kPW * (kPW / kRowWarps) <= sms;
}

int pcg_launch_count(const Sizes& s) { return 4 + (s.pcg_mode == 2 ? pcg_net_launch_count() : 0); }

int launch_pcg_blocks_only(const Sizes& s, const Dev& d, cudaStream_t st) {
  const PcgArgs a = pcg_args(s, d);
  const int64_t total = s.nsb * 36;
  const int blocks = static_cast<int>(std::min<int64_t>((total + kPT - 1) / kPT, 8192));
  k_pcg_scale<<<(s.n6 + 127) / 128, 128, 0, st>>>(a, d.ctrl);
  k_pcg_blocks<<<blocks > 0 ? blocks : 1, kPT, 0, st>>>(a, d.ctrl);
  return 2;
}

int launch_pcg(const Sizes& s, const Dev& d, cudaStream_t st) {
  return launch_pcg_blocks_only(s, d, st) + launch_pcg_scaled(s, d, st);
}

int launch_pcg_scaled(const Sizes& s, const Dev& d, cudaStream_t st) {
  const PcgArgs a = pcg_args(s, d);
  int n = 0;
  if (s.pcg_mode == 2) n += launch_pcg_net(s, d, st);
  k_pcg_precond<<<(s.nf + 3) / 4, 128, 0, st>>>(a, d.ctrl);
  ++n;
  cudaMemsetAsync(d.pcg_bar, 0, 4 * sizeof(unsigned), st);
  {
    cudaLaunchConfig_t cfg = {};
    const bool rows = s.pcg_row_max > 0;
    cfg.gridDim = dim3(rows ? s.pcg_grid * (kPW / kRowWarps) : s.pcg_grid);
    cfg.blockDim = dim3(rows ? 32 * kRowWarps : kPT);
    cfg.dynamicSmemBytes = rows ? rows_smem(s.nf, s.pcg_row_max) : 0;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (rows) cudaLaunchKernelEx(&cfg, k_pcg_rows, a, s.pcg_row_max, d.ctrl);
    else cudaLaunchKernelEx(&cfg, k_pcg_solve, a, d.ctrl);
    ++n;
  }
  return n;
}

}  // namespace sgba
