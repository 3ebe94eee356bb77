// sgba_dd.cuh -- float-float ("double-float", 48-bit significand) arithmetic
// on the FP32 pipes.
//
// GB300 issues FP32 FMAs at 128 per clock per SM but FP64 at about 2, so the
// FP64-class sums this solver needs (Hessian, Schur complement, costs) are
// carried as unevaluated pairs hi + lo of floats.  The building blocks are the
// error-free transformations of Knuth (TwoSum), Dekker (FastTwoSum) and the
// FMA-based TwoProduct, combined as in Hida, Li and Bailey's double-double
// library ("Algorithms for quad-double precision floating point arithmetic",
// ARITH 2001) but on float components.  Explicit _rn intrinsics keep the
// compiler from contracting or reassociating the transformations.
#pragma once

#include <cuda_runtime.h>

struct dd {
  float hi;
  float lo;
};

__host__ __device__ __forceinline__ dd dd_make(float hi, float lo) {
  dd r;
  r.hi = hi;
  r.lo = lo;
  return r;
}

// Knuth TwoSum: s + e == a + b exactly.
__device__ __forceinline__ dd dd_two_sum(float a, float b) {
  float s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return dd_make(s, e);
}

// Dekker FastTwoSum, valid when |a| >= |b| (or a == 0).
__device__ __forceinline__ dd dd_fast_two_sum(float a, float b) {
  float s = __fadd_rn(a, b);
  float e = __fsub_rn(b, __fsub_rn(s, a));
  return dd_make(s, e);
}

// TwoProduct with FMA: p + e == a * b exactly.
__device__ __forceinline__ dd dd_two_prod(float a, float b) {
  float p = __fmul_rn(a, b);
  float e = __fmaf_rn(a, b, -p);
  return dd_make(p, e);
}

__device__ __forceinline__ dd dd_neg(dd a) { return dd_make(-a.hi, -a.lo); }

// a + b, both double-float (accurate variant: TwoSum on both components).
__device__ __forceinline__ dd dd_add(dd a, dd b) {
  dd s = dd_two_sum(a.hi, b.hi);
  dd t = dd_two_sum(a.lo, b.lo);
  s.lo = __fadd_rn(s.lo, t.hi);
  s = dd_fast_two_sum(s.hi, s.lo);
  s.lo = __fadd_rn(s.lo, t.lo);
  return dd_fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ dd dd_sub(dd a, dd b) { return dd_add(a, dd_neg(b)); }

// a + b, b a float.
__device__ __forceinline__ dd dd_add_f(dd a, float b) {
  dd s = dd_two_sum(a.hi, b);
  s.lo = __fadd_rn(s.lo, a.lo);
  return dd_fast_two_sum(s.hi, s.lo);
}

// a * b
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
  dd p = dd_two_prod(a.hi, b.hi);
  p.lo = __fmaf_rn(a.hi, b.lo, p.lo);
  p.lo = __fmaf_rn(a.lo, b.hi, p.lo);
  return dd_fast_two_sum(p.hi, p.lo);
}

// a * b, b a float
__device__ __forceinline__ dd dd_mul_f(dd a, float b) {
  dd p = dd_two_prod(a.hi, b);
  p.lo = __fmaf_rn(a.lo, b, p.lo);
  return dd_fast_two_sum(p.hi, p.lo);
}

// c + a * b
__device__ __forceinline__ dd dd_fma(dd a, dd b, dd c) { return dd_add(c, dd_mul(a, b)); }

// a / b: long division with two float quotient digits and a correction
// (Hida-Li-Bailey "accurate" division restated for float components).
__device__ __forceinline__ dd dd_div(dd a, dd b) {
  float q1 = __fdiv_rn(a.hi, b.hi);
  dd r = dd_sub(a, dd_mul_f(b, q1));
  float q2 = __fdiv_rn(r.hi, b.hi);
  r = dd_sub(r, dd_mul_f(b, q2));
  float q3 = __fdiv_rn(r.hi, b.hi);
  dd q = dd_fast_two_sum(q1, q2);
  return dd_add_f(q, q3);
}

// sqrt(a) for a >= 0: one Newton correction of the float root, with the
// residual a - s*s formed exactly (Karp-Markstein style).
__device__ __forceinline__ dd dd_sqrt(dd a) {
  if (a.hi <= 0.0f) return dd_make(0.0f, 0.0f);
  float s = __fsqrt_rn(a.hi);
  dd s2 = dd_two_prod(s, s);
  dd e = dd_sub(a, s2);
  float corr = __fdiv_rn(e.hi, __fmul_rn(2.0f, s));
  return dd_fast_two_sum(s, corr);
}

// f64 <-> float-float.  The FP64 pipe of a GB300 SM sub-partition takes a warp
// 64 cycles per instruction, conversions between f32 and f64 included, so the
// plain forms (dd_from_double: narrow, widen, subtract, narrow; dd_to_double:
// widen, widen, add) cost 315 / 156 cycles in one warp and 2285 / 1179 with 32
// warps on an SM.  The same results (every bit, signs of zeros included) are
// formed from the mantissas with integer operations in 112 / 110 and 277 / 620
// cycles (dd_to_double keeps its one addition); exponents near the ends of the
// float range, infinities and NaN take the plain form.
__device__ __forceinline__ dd dd_from_double(double x) {
  const unsigned h = static_cast<unsigned>(__double2hiint(x)), l = static_cast<unsigned>(__double2loint(x));
  const unsigned e = (h >> 20) & 0x7ffu;
  if (e - 949u <= 200u) {  // 2^-74 .. 2^126: hi and lo are normal floats
    // hi = the upper 24 bits, to nearest even; lo = the other 29, signed
    const unsigned frac = (h << 3) | (l >> 29), rem = l & 0x1fffffffu, sgn = h & 0x80000000u;
    const unsigned up = rem + (frac & 1u) > 0x10000000u ? 1u : 0u;
    const int r = static_cast<int>(rem) - static_cast<int>(up << 29);
    const float lo = __int2float_rn(sgn ? -r : r) * __uint_as_float((e - 948u) << 23);
    return dd_make(__uint_as_float((((e - 896u) << 23) | (frac & 0x7fffffu)) + up | sgn), lo);
  }
  if (((h << 1) | l) == 0u) return dd_make(__uint_as_float(h), 0.0f);
  const float hi = __double2float_rn(x);
  return dd_make(hi, __double2float_rn(x - static_cast<double>(hi)));
}

__device__ __forceinline__ double dd_widen(float f) {
  const unsigned b = __float_as_uint(f), m = b & 0x7fffffffu, sgn = b & 0x80000000u;
  if (m - 0x00800000u < 0x7f000000u)  // normal
    return __hiloint2double(static_cast<int>(sgn | ((m >> 3) + 0x38000000u)), static_cast<int>(b << 29));
  return m == 0u ? __hiloint2double(static_cast<int>(sgn), 0) : static_cast<double>(f);
}

__device__ __forceinline__ double dd_to_double(dd a) { return dd_widen(a.hi) + dd_widen(a.lo); }

__device__ __forceinline__ dd dd_from_float(float x) { return dd_make(x, 0.0f); }

// Warp-level sum of a double-float (butterfly; every lane gets the total).
__device__ __forceinline__ dd dd_warp_sum(dd v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    dd o;
    o.hi = __shfl_xor_sync(0xffffffffu, v.hi, off);
    o.lo = __shfl_xor_sync(0xffffffffu, v.lo, off);
    v = dd_add(v, o);
  }
  return v;
}
