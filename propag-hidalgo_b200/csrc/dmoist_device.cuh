// Device side of the dmoist moisture model (crates/dmoist/src/lib.rs:55-715):
// the model's tables and per-cell functions, shared by the moisture pass
// (dmoist.cu) and the fused moisture + fire-behaviour pass (fire.cu).  Every
// file that includes it gets its own copy of the tables (global memory).  Float
// operations follow the reference's order; the including files are compiled
// without FMA contraction (explicit __fmaf_rn where the portable arctangent
// uses fused multiply-adds), so results equal the CPU restatement bit for bit.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace propag {

struct DmoistTables {
  int8_t hcb[6][21];
  uint8_t prob[4][9][18];
  int8_t shade[3][2][8][6];
  int8_t pp[2][4][6];
};

// The model's tables (lib.rs:197-262 base humidity index, daytime table;
// 272-453 ignition probability; 472-614 shading correction; 147-183
// precipitation effect), in DmoistTables order.
static __device__ const DmoistTables d_dm = {
    {
    {1, 2, 2, 3, 4, 5, 5, 6, 7, 8, 8, 8, 9, 9, 10, 11, 12, 12, 13, 13, 14},
    {1, 2, 2, 3, 4, 5, 5, 6, 7, 7, 7, 8, 9, 9, 10, 10, 11, 12, 13, 13, 13},
    {1, 2, 2, 3, 4, 5, 5, 6, 6, 7, 7, 8, 9, 9, 9, 10, 11, 12, 12, 12, 13},
    {1, 1, 2, 2, 3, 4, 5, 5, 6, 7, 7, 8, 8, 8, 9, 10, 10, 11, 12, 12, 13},
    {1, 1, 2, 2, 3, 4, 4, 5, 6, 7, 7, 8, 8, 8, 9, 10, 10, 11, 12, 12, 13},
    {1, 1, 2, 2, 3, 4, 4, 5, 6, 7, 7, 8, 8, 8, 9, 10, 10, 11, 12, 12, 12},
},
    {
    {{100, 100, 100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 30, 20, 20, 20, 10, 10},
     {100, 100, 90, 80, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 20, 10, 10, 10},
     {100, 100, 80, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 20, 10, 10, 10, 10}},
    {{100, 100, 100, 80, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 20, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 100, 80, 70, 60, 50, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 20, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 80, 70, 60, 50, 50, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10, 10}},
    {{100, 100, 90, 80, 70, 60, 50, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 100, 80, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 90, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 80, 70, 60, 50, 50, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10, 10}},
    {{100, 100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10},
     {100, 100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 20, 10, 10, 10},
     {100, 100, 80, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 50, 40, 30, 30, 30, 20, 20, 20, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 90, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 90, 70, 60, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10},
     {100, 80, 70, 60, 50, 50, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10, 10},
     {100, 80, 70, 60, 50, 40, 40, 30, 30, 20, 20, 20, 10, 10, 10, 10, 10, 10}},
},
    {
    {{{3, 1, 0, 0, 1, 3}, {4, 2, 1, 1, 2, 4}, {2, 1, 0, 0, 1, 4}, {2, 0, 0, 1, 3, 5},
      {3, 1, 0, 0, 1, 3}, {3, 1, 1, 1, 1, 3}, {3, 1, 0, 0, 1, 3}, {5, 3, 1, 0, 0, 2}},
     {{5, 4, 3, 3, 4, 5}, {5, 4, 3, 3, 4, 5}, {4, 4, 3, 4, 4, 5}, {4, 4, 3, 4, 4, 5},
      {4, 4, 3, 3, 4, 5}, {4, 4, 3, 3, 4, 5}, {5, 4, 3, 3, 4, 4}, {5, 4, 3, 3, 4, 4}}},
    {{{4, 2, 1, 1, 2, 4}, {4, 3, 3, 3, 3, 4}, {4, 2, 1, 1, 2, 4}, {3, 1, 1, 2, 4, 5},
      {4, 2, 1, 1, 2, 4}, {4, 2, 1, 1, 2, 4}, {4, 2, 1, 1, 2, 4}, {5, 4, 2, 1, 1, 3}},
     {{5, 5, 4, 4, 5, 5}, {5, 5, 4, 4, 5, 5}, {5, 4, 4, 4, 5, 5}, {5, 4, 4, 4, 5, 5},
      {5, 4, 4, 4, 4, 5}, {5, 4, 4, 4, 4, 5}, {5, 5, 4, 4, 4, 5}, {5, 5, 4, 4, 4, 5}}},
    {{{5, 4, 3, 3, 4, 5}, {5, 5, 5, 5, 5, 5}, {5, 4, 3, 3, 4, 5}, {5, 4, 3, 2, 5, 5},
      {5, 4, 3, 2, 4, 5}, {5, 3, 1, 1, 3, 5}, {5, 4, 3, 3, 4, 5}, {5, 5, 4, 2, 3, 5}},
     {{5, 5, 5, 5, 5, 5}, {5, 5, 5, 5, 5, 5}, {5, 5, 5, 5, 5, 5}, {5, 5, 5, 5, 5, 5},
      {5, 5, 5, 5, 5, 5}, {5, 5, 5, 5, 5, 5}, {5, 5, 5, 5, 5, 5}, {5, 5, 5, 5, 5, 5}}},
},
    {
    {{-1, -1, 0, 0, 0, 0}, {-1, 5, 1, 0, 0, 0}, {-1, 15, 5, 1, 0, 0}, {-1, 35, 15, 5, 1, 0}},
    {{-1, -1, -1, -1, 1, 0}, {-1, -1, -1, -1, 5, 1}, {-1, -1, -1, 15, 5, 1}, {-1, -1, 35, 15, 5, 1}},
},
};

// The tables as the kernels read them, in shared memory: ignition probability
// in tenths (its values are multiples of ten), and the quotients of a
// probability by itself corrected for precipitation (prob / dm_prob_precip,
// lib.rs:55-107), which take few values: row the precipitation class, column
// the probability in tenths; -1 where the corrected probability is zero.
struct DmoistShared {
  DmoistTables t;
  float ratio[5][11];
};

// Precipitation classes of the correction of the ignition probability.
__device__ __forceinline__ int dm_precip_class(float e) {
  if (e > 0.0f && e < 5.0f) return 1;
  if (e >= 5.0f && e < 15.0f) return 2;
  if (e >= 15.0f && e < 35.0f) return 3;
  return e >= 35.0f ? 4 : 0;
}
__device__ __forceinline__ float dm_prob_precip(float p, int cls) {
  const float a = cls == 0 ? 0.0f : cls == 1 ? -5.0f : -10.0f * (float)(cls - 1);
  const float v = p + a;
  return v < 0.0f ? 0.0f : (v > 100.0f ? 100.0f : v);
}

// Precipitation effect of day `offset` (mi: season row of the table).
__device__ __forceinline__ float dm_pp_effect(const DmoistTables &T, int mi, float pp, int offset) {
  if (pp > 0.0f) {
    const int pi = (pp >= 1.0f && pp < 5.0f) ? 0 : (pp >= 5.0f && pp < 15.0f) ? 1
                 : (pp >= 15.0f && pp < 35.0f) ? 2 : 3;
    const int e = T.pp[mi][pi][offset];
    if (e > -1) return (float)e;
  }
  return pp;
}

// floor(rh / 5) clamped to [0, 20] and 9 - ceil(t / 5) clamped to [0, 8]: the
// classes of the rounded product with 0.2f are those of the rounded quotient
// for every float (a test compares all of them).
__device__ __forceinline__ int dm_hcb(const DmoistTables &T, float t, float rh) {
  float hf = floorf(rh * 0.2f);
  hf = hf < 0.0f ? 0.0f : (hf > 20.0f ? 20.0f : hf);
  if (hf != hf) hf = 0.0f;  // NaN: class 0, as the reference's saturating cast
  int ti;
  if (t < 0.0f) ti = 0;
  else if (t >= 0.0f && t <= 9.0f) ti = 1;
  else if (t > 9.0f && t <= 20.0f) ti = 2;
  else if (t > 20.0f && t <= 31.0f) ti = 3;
  else if (t > 31.0f && t <= 42.0f) ti = 4;
  else ti = 5;
  return T.hcb[ti][(int)hf];
}

__device__ __forceinline__ float dm_shading(float cloud, int fuel) {
  float s = cloud * 0.75f;
  if (fuel >= 7 && fuel <= 12) s = s < 50.0f ? 75.0f : 100.0f;
  return s;
}

// Ignition probability in tenths; 0: none.
__device__ __forceinline__ int dm_prob(const DmoistTables &T, float t, float s, float hcs, int fuel) {
  if (fuel == 0) return 0;
  if (!(hcs > 0.0f && hcs < 18.0f)) return 0;
  const int si = (s >= 0.0f && s < 10.0f) ? 0 : (s >= 10.0f && s < 50.0f) ? 1
               : (s >= 50.0f && s < 90.0f) ? 2 : 3;
  float tf = 9.0f - ceilf(t * 0.2f);
  tf = tf < 0.0f ? 0.0f : (tf > 8.0f ? 8.0f : tf);
  if (tf != tf) tf = 0.0f;
  const int hci = (int)floorf(hcs) - 1;
  if (hci < 0) return 0;
  return T.prob[si][(int)tf][hci];
}

// What the shading correction takes from the hour and month alone: the
// table's season and hour columns, and whether the cloud cover counts.  (A
// month outside 1..12 has no season: DmoistRows::shaded.)
struct DmoistHour {
  int mi, hi;
  bool dark;  // fully shaded whatever the clouds
};
__device__ __forceinline__ DmoistHour dm_hour(int month, int hour) {
  DmoistHour h;
  h.mi = month >= 5 && month <= 8 ? 0 : (month >= 2 && month <= 4) || month == 9 || month == 10 ? 1 : 2;
  h.dark = !(hour >= 8 && hour <= 19);
  const int shown = hour >= 6 && hour < 8 ? 8 : hour >= 8 && hour <= 19 ? hour : 19;
  h.hi = (shown - 8) / 2;
  return h;
}

// The table's exposure row of a cell, or -1 (an aspect outside [0, 2 pi], or
// NaN, on a slope).  The reference compares aspect * 180 / pi with 45, 135,
// 225, 315 and 360 degrees and the slope's angle, atan(slope) * 180 / pi, with
// 30 degrees; each comparison is one with the first (last) float that passes it
// (a test compares the azimuths for every float, and the slopes for every float
// around 30 degrees and a spread of all).
__device__ __forceinline__ float dm_atan_pos(float y);
__device__ __forceinline__ int dm_exposure(float slope, float aspect) {
  constexpr float k45 = 0x1.921fb6p-1f, k135 = 0x1.2d97c8p+1f, k225 = 0x1.f6a7a4p+1f, k315 = 0x1.5fdbbep+2f;
  constexpr float kOver360 = 0x1.921fb8p+2f;     // the first aspect beyond 360 degrees
  constexpr float kSteepest30 = 0x1.279a74p-1f;  // the last slope not steeper than 30 degrees
  if (slope == 0.0f) return 4;
  int steep = slope <= kSteepest30 ? 0 : 1;
  if (slope < 0.0f) steep = dm_atan_pos(slope) * 180.0f / 3.14159274101257324f <= 30.0f ? 0 : 1;
  if (!(aspect >= 0.0f && aspect < kOver360)) return -1;
  const int quarter = aspect < k45 ? 0 : aspect < k135 ? 1 : aspect < k225 ? 2 : aspect < k315 ? 3 : 0;
  return 2 * quarter + steep;
}

// x / 15 and x / 9 from the rounded reciprocal of the constant and the product's
// residual by a fused multiply-add (Markstein 1990; Brisebarre, Muller and Raina
// 2004, on division by a divisor known in advance): the correctly rounded
// quotient for every finite float but -0, whose sign is lost (a test compares
// all of them).  The ends' differences are finite and not below 0.001.
__device__ __forceinline__ float dm_div15(float x) {
  const float r = 1.0f / 15.0f, q = x * r;
  return __fmaf_rn(__fmaf_rn(-15.0f, q, x), r, q);
}
__device__ __forceinline__ float dm_div9(float x) {
  const float r = 1.0f / 9.0f, q = x * r;
  return __fmaf_rn(__fmaf_rn(-9.0f, q, x), r, q);
}

// The 10-h interpolation between hours 6 and 15 (lib.rs:109-127): its two ends
// are the same for every hour of a cell.
struct DmoistEnds {
  float at6, at15;
  bool flat;
};
__device__ __forceinline__ DmoistEnds dm_ends(float m6, float m15) {
  DmoistEnds e;
  e.at6 = m15 + (0.4142f * (m6 - m15));
  e.at15 = m6 - (0.5571f * (m6 - m15));
  e.flat = fabsf(e.at6 - e.at15) < 0.001f;
  return e;
}
__device__ __forceinline__ float dm_by_10hr(int hour, float m, const DmoistEnds &e) {
  if (m == 0.0f) return 0.0f;
  if (e.flat) return e.at6 < 0.001f ? m : e.at6;
  if (hour >= 0 && hour < 6) return e.at15 + (dm_div15(e.at6 - e.at15) * (float)(hour + 15));
  if (hour >= 6 && hour < 15) return e.at6 + (dm_div9(e.at15 - e.at6) * (float)(hour - 6));
  if (hour >= 15 && hour < 24) return e.at15 + (dm_div15(e.at6 - e.at15) * (float)(hour - 15));
  return m;
}

// Portable arctangent of a non-negative ratio (the propagation code's
// series: octant reduction, odd series to u^19).
__device__ __forceinline__ float dm_atan_pos(float y) {
  const float mx = y > 1.0f ? y : 1.0f;
  const float mn = y > 1.0f ? 1.0f : y;
  const float t = mn / mx;
  float base = 0.0f, u = t;
  if (t > 0.414213562373095049f) {
    u = (t - 1.0f) / (t + 1.0f);
    base = 0.785398163397448309616f;
  }
  const float u2 = u * u;
  float p = __fmaf_rn(u2, 5.26315789e-2f, -5.88235294e-2f);
  p = __fmaf_rn(u2, p, 6.66666667e-2f);
  p = __fmaf_rn(u2, p, -7.69230769e-2f);
  p = __fmaf_rn(u2, p, 9.09090909e-2f);
  p = __fmaf_rn(u2, p, -1.11111111e-1f);
  p = __fmaf_rn(u2, p, 1.42857143e-1f);
  p = __fmaf_rn(u2, p, -2.00000000e-1f);
  p = __fmaf_rn(u2, p, 3.33333333e-1f);
  float a = __fmaf_rn(-(u * u2), p, u) + base;
  if (y > 1.0f) a = 1.57079632679489661923f - a;
  return a;
}

struct DmoistIn {
  const float *t, *rh, *cc;  // [24][n]
  const float *pp;           // [6][n]
  const float *slope, *aspect;
  const uint8_t *fuel;
};

// The rows of the weather rasters that a pass reads, and what depends on the
// hour and month alone; once per thread.
struct DmoistRows {
  const float *t[3], *rh[3], *cc[3];  // hours `hour`, 6 and 15
  const float *pp[6];
  DmoistHour h[3];
  int hour, season;  // season: row of the precipitation table
  bool shaded;       // the month has a shading correction (1..12)
};
__device__ __forceinline__ DmoistRows dmoist_rows(const DmoistIn &in, uint64_t n, int hour, int month) {
  DmoistRows r;
  const int hours[3] = {hour, 6, 15};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint64_t off = (uint64_t)hours[k] * n;
    r.t[k] = in.t + off;
    r.rh[k] = in.rh + off;
    r.cc[k] = in.cc + off;
    r.h[k] = dm_hour(month, hours[k]);
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) r.pp[d] = in.pp + (uint64_t)d * n;
  r.hour = hour;
  r.season = (month >= 4 && month <= 10) ? 0 : 1;
  r.shaded = month >= 1 && month <= 12;
  return r;
}

// Dead fuel moisture of cell i (percent): the 1-h moisture of the pass's hour
// and of hours 6 and 15, the 10-h class interpolated from those, the 100-h
// class from the 10-h values (lib.rs:109-127).  fuel, slope and aspect are the
// cell's (already loaded by the caller).
//
// Bound by instruction issue: the model took about 1 900 instructions a cell,
// most of them divisions, an arctangent that only decides on which side of 30
// degrees the slope lies, and work repeated for each of the three hours; with
// the fire behaviour it is 990 in all now.  1501 x 1403 cells of moisture and
// fire: 123 -> 85 us (tables copied from global instead of constant memory: 9
// of them).
template <typename Index>
__device__ __forceinline__ void dmoist_cell(const DmoistShared &T, const DmoistRows &in, Index i, int fuel,
                                            float slope, float aspect, float &d1, float &d10, float &d100) {
  float t[3], rh[3], cc[3], pp[6];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    t[k] = __ldg(in.t[k] + i);
    rh[k] = __ldg(in.rh[k] + i);
    cc[k] = __ldg(in.cc[k] + i);
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) pp[d] = __ldg(in.pp[d] + i);
  float ppmax = __int_as_float(0xff800000);  // -inf
#pragma unroll
  for (int d = 0; d < 6; ++d) ppmax = fmaxf(ppmax, dm_pp_effect(T.t, in.season, pp[d], d));
  const float *const ratio = T.ratio[dm_precip_class(ppmax)];
  const int oi = in.shaded ? dm_exposure(slope, aspect) : -1;
  float m1[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const DmoistHour &h = in.h[k];
    const float s = dm_shading(cc[k], fuel);
    const int shi = h.dark || !(s < 50.0f) ? 1 : 0;
    // a cell without an exposure row, or in a month the correction does not
    // know, has no corrected class (NaN in the reference): it takes neither a
    // probability nor the 30 % of a positive one
    float hcs = 0.0f;
    if (fuel != 0 && oi >= 0) hcs = (float)(dm_hcb(T.t, t[k], rh[k]) + T.t.shade[h.mi][shi][oi][h.hi]);
    const int p = dm_prob(T.t, t[k], s, hcs, fuel);
    const float q = ratio[p];
    m1[k] = q < 0.0f ? (hcs > 0.0f ? 30.0f : 0.0f) : q * hcs;
  }
  const DmoistEnds e = dm_ends(m1[1], m1[2]);
  const float m10h = dm_by_10hr(in.hour, m1[0], e);
  const float m10_6 = dm_by_10hr(6, m1[1], e);
  const float m10_15 = dm_by_10hr(15, m1[2], e);
  d1 = m1[0];
  d10 = m10h;
  d100 = dm_by_10hr(in.hour, m10h, dm_ends(m10_6, m10_15));
}

// The tables in shared memory, copied from global memory with coalesced loads
// (per-lane indices would serialise constant-memory reads); called by every
// thread of the block.
__device__ __forceinline__ void load_dmoist_tables(DmoistShared &T) {
  for (int k = threadIdx.x; k < (int)sizeof(DmoistTables); k += blockDim.x)
    reinterpret_cast<char *>(&T.t)[k] = reinterpret_cast<const char *>(&d_dm)[k];
  __syncthreads();
  uint8_t *const prob = &T.t.prob[0][0][0];
  for (int k = threadIdx.x; k < (int)sizeof(T.t.prob); k += blockDim.x) prob[k] = (uint8_t)(prob[k] / 10);
  for (int k = threadIdx.x; k < 55; k += blockDim.x) {
    const int cls = k / 11, p = k % 11;
    const float prob = 10.0f * (float)p, corrected = dm_prob_precip(prob, cls);
    T.ratio[cls][p] = corrected <= 0.0f ? -1.0f : __fdiv_rn(prob, corrected);
  }
  __syncthreads();
}

}  // namespace propag
