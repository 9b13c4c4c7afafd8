// Per-cell fire behaviour (Rothermel / BEHAVE) as an elementwise FP32 pass
// over structure-of-arrays rasters.
//
// Reference (paths relative to the reference project):
//   cuda_standard_simple_burn / cuda_standard_burn   crates/firelib/src/cuda.rs:7-95
//   Fuel::burn / burn_simple                         crates/firelib/src/firelib.rs:996-1030
//   rx_int_rbqig, eta_m                              firelib.rs:1031-1076
//   calculate_wind_dependent_vars, situations        firelib.rs:1078-1167
//   eccentricity, phi_slope, phi_wind                firelib.rs:1171-1188
//   Terrain::upslope                                 firelib.rs:400-409
//   Byram's intensity, flame length                  firelib.rs:424-441
//
// Layout and mapping: one cell per thread, grid-stride, so that every load
// and store of a warp is one coalesced run (4 bytes per lane, 1 for the fuel
// codes); 32-bit indices serve every grid below 2^32 cells.  The pass is bound
// by instruction issue and the warps in flight (360 instructions a cell; 516
// with double-float moisture sums for every cell and single-word table reads:
// 283 us at 4096^2, 215 now, each pass alone).  Four cells per thread with
// 128-bit loads measured slower (0.298 against 0.277 ms: four inlined copies of
// the cell code overflow the instruction cache), and so did loading a cell's inputs while the cell before
// it is computed (0.247 against 0.235 ms: 48 registers instead of 32 leave 40
// warps per SM instead of 64).  The fuel table sits in shared memory, a row's
// fields in the order they are read.  Compiled without automatic multiply-add
// contraction, so that the 3-field and 10-field instantiations round alike
// (contraction measured no faster).
//
// FP32 formulation.  The arithmetic is the reference's, rearranged where the
// float evaluation of the literal formula loses accuracy against double:
//   * the moisture sums are pre-folded per moisture class; the dead and live
//     sums and the live extinction moisture have more than float precision
//     (moist_sums), because they are subtracted from the moisture of
//     extinction, where float cancellation would dominate the error;
//   * eta_m = 1 - 2.59 rt + 5.11 rt^2 - 3.52 rt^3 is evaluated in
//     u = 1 - rt = (mext - moist) / mext as u (2.93 - 5.45 u + 3.52 u^2),
//     the same cubic expanded at rt = 1 where it vanishes;
//   * the cross-slope direction uses atan2(|y|, |x|) instead of
//     asin(|y| / hypot(x, y)) (same angle, no loss near 90 degrees);
//   * the cross-slope vector is summed in phi units (the reference's rate
//     vectors divided by speed0 > 0), so phi_ew2 is its length instead of
//     (speed0 + rv) / speed0 - 1;
//   * eccentricity sqrt(lw^2 - 1) / lw with lw = 1 + a is sqrt(a (2 + a)) / (1 + a);
//   * pi and 2 pi are added as float pairs (hi + lo).
#include <cuda_runtime.h>

#include <cstdint>

#include "catalog.hpp"
#include "dmoist_device.cuh"
#include "moist_sums.cuh"

namespace propag {

constexpr float kSmidgenF = 1e-6f;  // SMIDGEN, crates/firelib/src/f32.rs:5
constexpr float kPiHi = 3.14159274101257324f, kPiLo = -8.74227766e-8f;
constexpr float kTwoPiHi = 6.28318548202514648f, kTwoPiLo = -1.74845553e-7f;
// unit conversions (crates/firelib/src/units.rs:28-30: foot 0.3048 m,
// BTU 1054.35 J)
constexpr float kFpmToMps = 0.00508f;             // 0.3048 / 60
constexpr float kMpsToFpm = 196.850393700787402f; // 60 / 0.3048
constexpr float kRxToSI = 189.146876418865f;      // BTU/ft^2/min -> W/m^2
constexpr float kHpuaToSI = 11348.8125851319f;    // BTU/ft^2 -> J/m^2
constexpr float kByramsToSI = 3459.15354330709f;  // BTU/ft/s -> W/m
constexpr float kFootToM = 0.3048f;

// The fuel table in global memory: every block copies it to shared memory with
// coalesced loads (per-lane indices would serialise constant-memory reads).
__device__ FuelConst d_catalog[kMaxFuels];

struct FireOut {
  float rx_int, speed0, hpua, phi_eff_wind, speed_max, azimuth_max, eccentricity,
      residence_time, byrams, flame;
};

// 1 - rt of the dead fuel, (mext - dead_moist) / mext, as the product with the
// model's mext_rcp: an operation of its own, whose relative error is at most
// 2^-22 for the reciprocal (CUDA's bound for __fdividef is 2 ulp) and 2^-24 for
// the product.  A test holds it to that and compares it with __fdividef(dead,
// mext).
__device__ __forceinline__ float dead_ratio(const FuelConst &F, float dead) { return dead * F.mext_rcp; }

// eta_m (firelib.rs:1060-1076) with rt = moist / mext, as
// u (2.93 - 5.45 u + 3.52 u^2), u = 1 - rt = (mext - moist) / mext.
__device__ __forceinline__ float eta_of(float u) { return u * fmaf(u, fmaf(u, 3.52f, -5.45f), 2.93f); }

// x^y for x >= 0 (0^y = 0 for y > 0) as 2^(y log2 x): about 1e-6 relative
// (|y log2 x| < 30 here), well inside the fields' 1e-5 budget, at a fraction
// of powf's cost (powf keeps extended precision for < 1 ulp).
__device__ __forceinline__ float pow_pos(float x, float y) { return exp2f(y * log2f(x)); }

__device__ __forceinline__ float dot5(const float *c, const float m[5]) {
  float s = c[0] * m[0];
  s = fmaf(c[1], m[1], s);
  s = fmaf(c[2], m[2], s);
  s = fmaf(c[3], m[3], s);
  return fmaf(c[4], m[4], s);
}

template <bool kFull>
__device__ __forceinline__ void burn_cell(const FuelConst &F, const float m[5], float ws,
                                          float waz, float slope, float aspect, FireOut &o) {
  // rx_int_rbqig
  const float rbqig = F.R0 + dot5(F.R, m);
  const Moist w = moist_sums(F, m);
  // not positive: life_moist >= life_mext.  __fdividef: operands in [2^-126, 2^126]
  const float eta_dead = w.dead > 0.0f ? eta_of(dead_ratio(F, w.dead)) : 0.0f;
  const float eta_live = w.live > 0.0f ? eta_of(__fdividef(w.live, w.lmext)) : 0.0f;
  const float rx = fmaf(F.rx_alive, eta_live, F.rx_dead * eta_dead);
  const float speed0 = __fdividef(rx * F.flux_ratio, rbqig);

  // calculate_wind_dependent_vars
  const float phi_slope = F.slope_k * slope * slope;
  const float ws_fpm = ws * kMpsToFpm;
  const float phi_wind = F.wind_k * pow_pos(ws_fpm, F.wind_b);
  const float phi_ew = phi_slope + phi_wind;
  const float upslope = aspect >= kPiHi ? (aspect - kPiHi) - kPiLo : (aspect + kPiHi) + kPiLo;
  const float max_wind = 0.9f * rx;

  float pew = phi_ew, ew = 0.0f, smax = 0.0f, az = 0.0f;
  bool limit = true;
  if (speed0 < kSmidgenF) {  // NoSpread
    limit = false;
  } else if (phi_ew < kSmidgenF) {  // NoSlopeNoWind
    smax = speed0;
    limit = false;
  } else if (slope < kSmidgenF) {  // WindNoSlope
    ew = ws_fpm;
    smax = speed0 * (1.0f + phi_ew);
    az = waz;
  } else if (ws < kSmidgenF || fabsf(upslope - waz) < kSmidgenF) {  // SlopeNoWind, UpSlope
    ew = pow_pos(phi_ew * F.wind_e, F.wind_b_inv);
    smax = speed0 * (1.0f + phi_ew);
    az = upslope;
  } else {  // CrossSlope
    // The reference sums the rate vectors speed0 * phi; the common factor
    // speed0 > 0 is kept out: (x, y) below are those vectors / speed0, the
    // direction and quadrant are unchanged and phi_ew2 = |(x, y)|.
    const float split = upslope <= waz ? waz - upslope : ((kTwoPiHi - upslope) + waz) + kTwoPiLo;
    // the same angle in [-pi, pi], where the fast sine and cosine are
    // accurate to 2^-21.4 absolute (the vector components are then good to
    // ~4e-7 of phi_wind, inside the fields' 1e-5 budget)
    const float red = split > kPiHi ? (split - kTwoPiHi) - kTwoPiLo : split;
    float sn, cs;
    __sincosf(red, &sn, &cs);
    const float x = fmaf(phi_wind, cs, phi_slope);
    const float y = phi_wind * sn;
    pew = sqrtf(fmaf(x, x, y * y));  // phi values far below 1e18: no overflow to guard
    smax = speed0 * (1.0f + pew);
    ew = pow_pos(pew * F.wind_e, F.wind_b_inv);
    const float al = atan2f(fabsf(y), fabsf(x));
    float split2;
    if (x >= 0.0f && y >= 0.0f) split2 = al;
    else if (x >= 0.0f) split2 = (kTwoPiHi - al) + kTwoPiLo;
    else if (y >= 0.0f) split2 = (kPiHi - al) + kPiLo;
    else split2 = (kPiHi + al) + kPiLo;
    az = upslope + split2;
    if (az > kTwoPiHi) az = (az - kTwoPiHi) - kTwoPiLo;
  }
  if (limit && ew > max_wind) {  // check_wind_limit
    pew = F.wind_k * pow_pos(max_wind, F.wind_b);
    ew = max_wind;
    smax = speed0 * (1.0f + pew);
  }
  const float a = 0.002840909f * ew;
  o.speed_max = smax * kFpmToMps;
  o.azimuth_max = az;
  o.eccentricity = __fdividef(sqrtf(a * (2.0f + a)), 1.0f + a);
  if (kFull) {  // the remaining FireCuda fields, Byram and flame
    o.rx_int = rx * kRxToSI;
    o.speed0 = speed0 * kFpmToMps;
    o.hpua = rx * F.residence_time * kHpuaToSI;
    o.phi_eff_wind = pew;
    o.residence_time = F.residence_time * 60.0f;
    const float byrams = F.residence_time * smax * rx * (1.0f / 60.0f);
    o.byrams = byrams * kByramsToSI;
    o.flame = byrams > kSmidgenF ? 0.45f * pow_pos(byrams, 0.46f) * kFootToM : 0.0f;
  }
}

struct Inputs {
  const uint8_t *fuel;
  const float *m[5];
  const float *ws, *waz, *slope, *aspect;
};
struct Outputs {
  float *f[10];  // PropagFireFields order
};

// kFull: every field whose output is given; else the three the propagation
// needs (the 3-field entry point passes only those).
template <bool kFull, typename Index>
__device__ __forceinline__ void store_cell(const Outputs &out, Index i, const FireOut &o) {
  const float v[10] = {o.rx_int, o.speed0, o.hpua, o.phi_eff_wind, o.speed_max,
                       o.azimuth_max, o.eccentricity, o.residence_time, o.byrams, o.flame};
#pragma unroll
  for (int k = 0; k < 10; ++k)
    if ((kFull || (k >= 4 && k <= 6)) && out.f[k]) out.f[k][i] = v[k];
}

// Shared-memory copy of the fuel table, rows kCatStride words apart: a
// multiple of four (16-byte loads) whose quads 11 f mod 8 lie in different
// banks for any eight models in a row.
constexpr int kCatStride = 44;
static_assert(sizeof(FuelConst) / 4 <= kCatStride, "a FuelConst fits a table row");

__device__ __forceinline__ void load_catalog(float *cat) {
  const float *src = reinterpret_cast<const float *>(d_catalog);
  constexpr int kWords = (int)(sizeof(FuelConst) / 4);
  for (int t = threadIdx.x; t < kMaxFuels * kWords; t += blockDim.x)
    cat[(t / kWords) * kCatStride + t % kWords] = src[t];
  __syncthreads();
  if (threadIdx.x < kMaxFuels) {
    FuelConst *const f = reinterpret_cast<FuelConst *>(cat + threadIdx.x * kCatStride);
    f->mext_rcp = __fdividef(1.0f, f->mext_f);
  }
  __syncthreads();
}

__device__ __forceinline__ const FuelConst &fuel_row(const float *cat, uint32_t code) {
  return *reinterpret_cast<const FuelConst *>(cat + code * kCatStride);
}

template <bool kFull, typename Index>
__device__ __forceinline__ void one_cell(const float *cat, const Inputs &in, const Outputs &out,
                                         Index i) {
  const uint8_t code = __ldg(in.fuel + i);
  FireOut o{};
  if (code < kMaxFuels && fuel_row(cat, code).has_fire != 0.0f) {
    const float m[5] = {__ldg(in.m[0] + i), __ldg(in.m[1] + i), __ldg(in.m[2] + i), __ldg(in.m[3] + i),
                        __ldg(in.m[4] + i)};
    burn_cell<kFull>(fuel_row(cat, code), m, __ldg(in.ws + i), __ldg(in.waz + i),
                     __ldg(in.slope + i), __ldg(in.aspect + i), o);
  }
  store_cell<kFull>(out, i, o);
}

// One cell per thread, grid-stride, cells [first, n): every load and store is
// coalesced (4 or 1 consecutive bytes per lane).  kFull: all ten fields; else
// the three the propagation needs (the shared fields are the same
// operations, so both give the same values for them).
// Index: uint32_t when n + the grid's threads fit in 32 bits (cheaper
// address arithmetic), else uint64_t.  Six CTAs an SM: 40 registers (44 to 47
// without the bound: 240 us against 225 at 4096^2 in one wave of CTAs; 32 for
// eight CTAs: 230).
template <bool kFull, typename Index>
__global__ void __launch_bounds__(256, 6) fire_kernel(Inputs in, Outputs out, Index first, Index n) {
  __shared__ __align__(16) float cat[kMaxFuels * kCatStride];
  load_catalog(cat);
  const Index stride = (Index)gridDim.x * blockDim.x;
  for (Index i = first + (Index)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    one_cell<kFull>(cat, in, out, i);
}

// Dead fuel moisture and fire behaviour in one pass (no d1/d10/d100 rasters
// in between): per cell the dmoist model at `hour` from the cell's weather
// (dmoist_cell, percent values scaled to fractions as the moisture pass's
// scale 0.01 does), then the three fields the propagation needs.  The same
// operations as the moisture pass followed by fire_kernel<false>, so the
// same bits.  Cells without fire skip the moisture model (their outputs are
// 0 either way).
template <typename Index>
__global__ void __launch_bounds__(256) fire_weather_kernel(DmoistIn win, int hour, int month,
                                                           Inputs in, Outputs out, Index n) {
  __shared__ __align__(16) float cat[kMaxFuels * kCatStride];
  __shared__ DmoistShared T;
  load_dmoist_tables(T);
  load_catalog(cat);
  const DmoistRows rows = dmoist_rows(win, (uint64_t)n, hour, month);
  const Index stride = (Index)gridDim.x * blockDim.x;
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint8_t code = __ldg(in.fuel + i);
    FireOut o{};
    if (code < kMaxFuels && fuel_row(cat, code).has_fire != 0.0f) {
      const float slope = __ldg(in.slope + i), aspect = __ldg(in.aspect + i);
      float m1, m10, m100;
      dmoist_cell(T, rows, i, code, slope, aspect, m1, m10, m100);
      const float m[5] = {m1 * 0.01f, m10 * 0.01f, m100 * 0.01f, __ldg(in.m[3] + i), __ldg(in.m[4] + i)};
      burn_cell<false>(fuel_row(cat, code), m, __ldg(in.ws + i), __ldg(in.waz + i), slope, aspect, o);
    }
    store_cell<false>(out, i, o);
  }
}

// CTAs of a fire kernel resident per SM (registers limit it).
template <typename K>
static int ctas_per_sm(K kernel, int threads) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) != cudaSuccess || n < 1)
    n = 1;
  return n;
}

// As many CTAs as are resident at once, each striding over an equal share: a
// small grid's table copies and partial last wave would cost more than they
// balance.  Up to four times as many when a thread still has eight cells to
// compute: equal shares take unequal time (patches that do not burn, divergent
// cells), and 4096^2 cells ran 231 us in one wave, with the SMs' warps active
// 80 % of the time, 215 in four, 219 in sixteen; 1.9 M cells 37 us in one, 43 in
// sixteen.
static unsigned grid_for(uint64_t items, int threads, int sm_count, int per_sm) {
  const uint64_t wave = (uint64_t)sm_count * (uint64_t)per_sm;
  const uint64_t waves = items / (wave * (uint64_t)threads * 8);
  const uint64_t cap = wave * (waves < 1 ? 1 : waves > 4 ? 4 : waves);
  uint64_t blocks = (items + threads - 1) / threads;
  if (blocks > cap) blocks = cap;
  return blocks ? (unsigned)blocks : 1u;
}

template <bool kFull, typename Index>
static cudaError_t launch_fire_t(const Inputs &in, const Outputs &out, uint64_t n, int sm_count,
                                 int threads, cudaStream_t stream) {
  auto k1 = fire_kernel<kFull, Index>;
  k1<<<grid_for(n, threads, sm_count, ctas_per_sm(k1, threads)), threads, 0, stream>>>(in, out, (Index)0,
                                                                                    (Index)n);
  return cudaGetLastError();
}

// For the test of dead_ratio: it, __fdividef and the divisor, for model[i] and dead[i].
__global__ void dead_ratio_kernel(uint64_t n, const int32_t *model, const float *dead, float *product,
                                  float *quotient, float *mext) {
  __shared__ __align__(16) float cat[kMaxFuels * kCatStride];
  load_catalog(cat);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const FuelConst &F = fuel_row(cat, (uint32_t)model[i] < kMaxFuels ? model[i] : 0);
    product[i] = dead_ratio(F, dead[i]);
    quotient[i] = __fdividef(dead[i], F.mext_f);
    mext[i] = F.mext_f;
  }
}

cudaError_t launch_dead_ratio(uint64_t n, const int32_t *model, const float *dead, float *product, float *quotient,
                              float *mext, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  dead_ratio_kernel<<<256, 256, 0, stream>>>(n, model, dead, product, quotient, mext);
  return cudaGetLastError();
}

// ---- host-side launchers (called from api.cpp) ------------------------------
cudaError_t upload_catalog() {
  FuelConst table[kMaxFuels];
  if (!build_catalog_table(table)) return cudaErrorInvalidValue;
  return cudaMemcpyToSymbol(d_catalog, table, sizeof(table));
}

cudaError_t launch_fire(bool full, uint64_t n, const uint8_t *fuel, const float *const m[5],
                        const float *ws, const float *waz, const float *slope,
                        const float *aspect, float *const outs[10], int sm_count,
                        cudaStream_t stream) {
  Inputs in{fuel, {m[0], m[1], m[2], m[3], m[4]}, ws, waz, slope, aspect};
  Outputs out{};
  for (int k = 0; k < 10; ++k) out.f[k] = outs[k];
  if (n == 0) return cudaSuccess;
  const int threads = 256;
  // 32-bit indices while the last index plus one grid stride (four waves) stays below 2^32
  const bool narrow = n + 4 * (uint64_t)sm_count * 8 * threads < (1ull << 32);
  if (full)
    return narrow ? launch_fire_t<true, uint32_t>(in, out, n, sm_count, threads, stream)
                  : launch_fire_t<true, uint64_t>(in, out, n, sm_count, threads, stream);
  return narrow ? launch_fire_t<false, uint32_t>(in, out, n, sm_count, threads, stream)
                : launch_fire_t<false, uint64_t>(in, out, n, sm_count, threads, stream);
}

cudaError_t launch_fire_weather(uint64_t n, int hour, int month, const float *t, const float *rh,
                                const float *cc, const float *pp, const uint8_t *fuel,
                                const float *herb, const float *wood, const float *ws,
                                const float *waz, const float *slope, const float *aspect,
                                float *speed_max, float *azimuth_max, float *eccentricity,
                                int sm_count, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  DmoistIn win{t, rh, cc, pp, slope, aspect, fuel};
  Inputs in{fuel, {nullptr, nullptr, nullptr, herb, wood}, ws, waz, slope, aspect};
  Outputs out{};
  out.f[4] = speed_max;
  out.f[5] = azimuth_max;
  out.f[6] = eccentricity;
  const int threads = 256;
  const bool narrow = n + 4 * (uint64_t)sm_count * 8 * threads < (1ull << 32);
  if (narrow) {
    auto k = fire_weather_kernel<uint32_t>;
    k<<<grid_for(n, threads, sm_count, ctas_per_sm(k, threads)), threads, 0, stream>>>(
        win, hour, month, in, out, (uint32_t)n);
  } else {
    auto k = fire_weather_kernel<uint64_t>;
    k<<<grid_for(n, threads, sm_count, ctas_per_sm(k, threads)), threads, 0, stream>>>(
        win, hour, month, in, out, (uint64_t)n);
  }
  return cudaGetLastError();
}

}  // namespace propag
