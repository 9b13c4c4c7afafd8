// The moisture sums of the fire-behaviour pass (firelib.rs:1031-1076).
//
// The numerators and the denominator of 1 - rt (eta_m below): mext - dead_moist,
// live_mext - live_moist and live_mext, rounded to float from double-float
// values (hi + lo, |lo| <= ulp(hi) / 2), whose relative error is at most 2^-42.5
// of the sum of the terms' magnitudes.
//
// They are worked out in double (eight multiply-adds instead of about 150 float
// operations), which rounds to the same float unless the value lies within
// that error of a point where the rounding changes; then (none to one cell in a
// thousand by model, 0.04 % over all of them on ordinary moistures) the
// double-float sums decide, so that the results are the double-float ones bit
// for bit: a propagation depends on its fire fields to the last bit.  (4096^2 in
// 215 us; without the check 207, with the double-float sums inlined 229, and with
// those cells put off to the thread's end 1.09 times as long.)
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "catalog.hpp"

#if !defined(__CUDACC__)  // host code (built without contraction): the same operations
#define __device__
#define __noinline__ __attribute__((noinline))
#define __forceinline__ inline
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline int __double2loint(double v) {
  uint64_t b;
  std::memcpy(&b, &v, 8);
  return (int)(uint32_t)b;
}
#endif

namespace propag {

struct Moist {
  float dead, live, lmext;
};

struct DF {
  float hi, lo;
};
// Error-free sum of two floats (Knuth's two-sum).
__device__ __forceinline__ DF two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return DF{s, e};
}
__device__ __forceinline__ DF df_of(double v) {
  const float hi = (float)v;
  return DF{hi, (float)(v - (double)hi)};
}
// sum of c[k] * m[k]: exact products (fma) and sums (two-sum).
template <int N>
__device__ __forceinline__ DF dot_df(const double *c, const float *m) {
  float hi = 0.0f, lo = 0.0f;
  for (int k = 0; k < N; ++k) {
    const DF w = df_of(c[k]);
    const float p = __fmul_rn(w.hi, m[k]);
    const float pe = __fmaf_rn(w.hi, m[k], -p);
    const DF s = two_sum(hi, p);
    hi = s.hi;
    lo = __fadd_rn(lo, __fadd_rn(s.lo, __fmaf_rn(w.lo, m[k], pe)));
  }
  return two_sum(hi, lo);
}
__device__ __forceinline__ DF df_sub(DF a, DF b) {
  const DF s = two_sum(a.hi, -b.hi);
  return two_sum(s.hi, __fadd_rn(s.lo, __fsub_rn(a.lo, b.lo)));
}
__device__ __noinline__ Moist moist_df(const FuelConst &F, float m0, float m1, float m2, float m3, float m4) {
  const float m[5] = {m0, m1, m2, m3, m4};
  const DF mext = df_of(F.mext);
  const DF dead = df_sub(mext, dot_df<3>(F.A, m));
  DF lmext{0.0f, 0.0f};
  if (F.has_live != 0.0f) {
    lmext = df_sub(df_of(F.LM0), dot_df<3>(F.LM, m));
    if (!(df_sub(lmext, mext).hi > 0.0f)) lmext = mext;  // max(live_mext, mext)
  }
  const DF live = df_sub(lmext, dot_df<2>(F.B, m + kHerb));
  return Moist{dead.hi + dead.lo, live.hi + live.lo, lmext.hi + lmext.lo};
}

// Whether v and every value nearer to it than 2^(kTol - 53) |v| round to the same
// float: v's distance from the midpoint of two floats is more than 2^kTol units
// of its own last place (2^(E-52) for |v| in [2^E, 2^(E+1))).  The midpoint has
// the low 29 of the mantissa's 52 bits at 2^28.
template <int kTol>
__device__ __forceinline__ bool rounds_surely(double v) {
  return ((uint32_t)__double2loint(v) << 3) + 0x80000000u + (8u << kTol) > (16u << kTol);
}

// The sums in double; false when they may not round as the double-float ones do.
__device__ __forceinline__ bool moist_double(const FuelConst &F, const float *m, Moist &r) {
  const double m0 = (double)m[0], m1 = (double)m[1], m2 = (double)m[2];
  const double dead = __fma_rn(-F.A[2], m2, __fma_rn(-F.A[1], m1, __fma_rn(-F.A[0], m0, F.mext)));
  r = Moist{(float)dead, 0.0f, 0.0f};
  // For moistures that are not negative the terms' magnitudes S sum to at most
  // 2 mext where dead is positive (its rounding does not matter where it is
  // not), so S <= 8 dead above dead_min = mext / 4, and the error 2^-42 S is at
  // most 2^(14 - 53) dead.  (dead_exact: a model whose sum is exact either way,
  // and often lies halfway between two floats.)
  bool sure = (fminf(fminf(m[0], m[1]), m[2]) >= 0.0f) & (fabsf(r.dead) > F.dead_min) &
              (rounds_surely<14>(dead) | (F.dead_exact != 0.0f));
  if (F.has_live != 0.0f) {
    const double raw = __fma_rn(-F.LM[2], m2, __fma_rn(-F.LM[1], m1, __fma_rn(-F.LM[0], m0, F.LM0)));
    const double lmext = raw > F.mext ? raw : F.mext;  // max(live_mext, mext)
    const double live = __fma_rn(-F.B[1], (double)m[4], __fma_rn(-F.B[0], (double)m[3], lmext));
    const float raw_f = (float)raw;
    r.live = (float)live;
    r.lmext = fmaxf(raw_f, F.mext_f);  // the float of lmext
    // raw clearly the larger of the two, and large enough, or clearly the
    // smaller (then lmext is mext itself).  S is at most 2 (LM0 + mext), 32 times
    // live_min = (LM0 + mext) / 16, and the error of two sums 2^-41 S
    sure = sure & (fminf(m[3], m[4]) >= 0.0f) & (((raw_f > F.live_above) & rounds_surely<17>(raw)) | (raw_f < F.live_below)) &
           (fabsf(r.live) > F.live_min) & rounds_surely<17>(live);
  }
  return sure;
}
__device__ __forceinline__ Moist moist_sums(const FuelConst &F, const float *m) {
  Moist r;
  return moist_double(F, m, r) ? r : moist_df(F, m[0], m[1], m[2], m[3], m[4]);
}

}  // namespace propag
