// The line-of-sight walk of propag.h:91-135 in closed form, column by column.
//
// The walk from one cell to another, |dx| and |dy| cells away, merges two
// arithmetic progressions of crossing times, i / |dx| and j / |dy|, each
// accumulated in float (start 1 / |d|, step + 1 / |d|), and takes a diagonal
// step when two crossings are closer than 1e-9.  Let P be the larger offset
// and Q the smaller one.  For P, Q <= kColumnsMax the accumulated values stay
// within 2 * 128 * 2^-24 = 1.6e-5 of the exact ones, while crossings that do
// not coincide exactly are at least 1 / (P Q) >= 6.2e-5 apart: the float order
// of two crossings is the exact order unless they coincide, which happens at
// the columns c with c Q a multiple of P.  There the accumulated values
// decide (kinds below).  So the cells of column c (the c-th step along the
// longer axis) follow from integer arithmetic and, at coinciding crossings,
// two accumulated values; at most two cells of a column are visited.  A test
// checks every offset against the step-by-step walk.
#pragma once

#include <cstdint>

#if !defined(__CUDACC__) && !defined(__device__)  // host code: plain functions
#define __device__
#define __forceinline__ inline
#endif
#if defined(__CUDACC__)
#define PG_HOST_DEVICE __host__ __device__
#else
#define PG_HOST_DEVICE
#endif

namespace propag {

constexpr int kColumnsMax = 127;
// Accumulated crossing times: T(n, i) (i steps of 1 / n) at n (n - 1) / 2 + i - 1.
constexpr int kCrossTableLen = kColumnsMax * (kColumnsMax + 1) / 2;

PG_HOST_DEVICE inline int cross_at(int n, int i) { return n * (n - 1) / 2 + i - 1; }

// Rows crossed strictly before the c-th crossing of the longer axis, and
// whether a row crossing coincides with it.  inv_p is 1 / P rounded to float:
// (c Q - 1/2) / P is at least 1 / (2 P) away from an integer, far more than
// the float product's error.
__device__ __forceinline__ int rows_before(int P, int Q, int c, float inv_p, bool &tie) {
  const int u = c * Q;
  const int j = (int)(((float)u - 0.5f) * inv_p);
  tie = u == (j + 1) * P;
  return j;
}

// At a coinciding crossing (column c, row j + 1): 0 the column is entered
// first, 1 a diagonal step, 2 the row is crossed first.
__device__ __forceinline__ int cross_kind(const float *table, int P, int Q, int c, int j) {
  const float d = table[cross_at(P, c)] - table[cross_at(Q, j + 1)];
  // 9.99999972e-10: the largest float below 1e-9
  return d < -9.99999972e-10f ? 0 : d > 9.99999972e-10f ? 2 : 1;
}

// The cells of column c: rows jin .. jout (the same, or two), and whether the
// column was entered by a diagonal step.
__device__ __forceinline__ void walk_column(const float *table, int P, int Q, int c, float inv_p, int &jin,
                                            int &jout, bool &diag) {
  bool t0, t1;
  const int a = rows_before(P, Q, c, inv_p, t0);
  const int b = rows_before(P, Q, c + 1, inv_p, t1);
  jin = a;
  diag = false;
  if (t0) {
    const int k = cross_kind(table, P, Q, c, a);
    jin = a + (k != 0);
    diag = k == 1;
  }
  if (c == P)
    jout = Q;
  else
    jout = t1 && cross_kind(table, P, Q, c + 1, b) == 2 ? b + 1 : b;
}

}  // namespace propag
