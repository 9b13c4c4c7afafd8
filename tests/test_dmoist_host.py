"""The dmoist model's device code (csrc/dmoist_device.cuh) compiled for the
host, against the CPU restatement of the reference (crates/dmoist/src/
lib.rs:55-715): equal bit for bit in every month a caller can pass, the ones
outside 1..12 included, for which the reference has no shading correction (the
corrected humidity class is NaN there, and every moisture zero).  What it
computes another way than the model's formulas -- divisions by constants,
classes, limits of the exposures -- is compared with them float by float."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "propag-hidalgo_b200", "csrc")

# the CUDA built-ins that the header uses, for one thread
SHIM = r"""
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __ldg(p) (*(p))
struct Dim { unsigned x; };
static const Dim threadIdx{0}, blockDim{1};
static inline void __syncthreads() {}
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
"""

SOURCE = r"""
#include "dmoist_device.cuh"
using namespace propag;
extern "C" void cells(long n, int hour, int month, const float *t, const float *rh, const float *cc, const float *slope,
                      const float *aspect, const uint8_t *fuel, const float *pp, float *d1, float *d10, float *d100) {
  static DmoistShared T;
  load_dmoist_tables(T);
  const DmoistRows rows = dmoist_rows(DmoistIn{t, rh, cc, pp, slope, aspect, fuel}, (uint64_t)n, hour, month);
  for (long i = 0; i < n; ++i) dmoist_cell(T, rows, i, fuel[i], slope[i], aspect[i], d1[i], d10[i], d100[i]);
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("dmoist")
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "m.cpp").write_text(SOURCE)
    so = d / "m.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-shared", "-fPIC", "-I" + str(d),
                    "-I" + CSRC, str(d / "m.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    return dict(temperature=rng.uniform(-10, 48, (24, n)).astype(np.float32),
                humidity=rng.uniform(0, 100, (24, n)).astype(np.float32),
                cloud_cover=rng.uniform(0, 100, (24, n)).astype(np.float32),
                slope=(rng.uniform(0, 1.6, n) * (rng.random(n) < 0.9)).astype(np.float32),
                aspect=rng.uniform(-0.5, 7.0, n).astype(np.float32),
                fuel_code=rng.integers(0, 16, n).astype(np.uint8),
                precipitation=(rng.uniform(0, 50, (6, n)) * (rng.random((6, n)) < 0.4)).astype(np.float32))


@pytest.mark.parametrize("month", list(range(1, 13)) + [0, 13, -1, 1 << 30])
def test_every_month(model, oracle, month):
    n = 3001
    for hour in (0, 6, 7, 8, 14, 19, 23):
        x = _inputs(n, 24 * (month % 100) + hour)
        got = [np.zeros(n, np.float32) for _ in range(3)]
        model.cells(C.c_long(n), C.c_int(hour), C.c_int(month), *[_ptr(x[k]) for k in x], *[_ptr(g) for g in got])
        want = oracle.dmoist_cells(hour, month, *[x[k] for k in x])
        for g, w in zip(got, want):
            assert np.array_equal(g.view(np.uint32), w.view(np.uint32)), hour
        if not 1 <= month <= 12:
            assert not np.any(got[0])


# Each function returns the number of floats for which the device code differs
# from the model's formula.
EXHAUSTIVE = r"""
#include "dmoist_device.cuh"
using namespace propag;
static inline float as_float(uint32_t b) { float f; std::memcpy(&f, &b, 4); return f; }
static inline uint32_t bits(float f) { uint32_t b; std::memcpy(&b, &f, 4); return b; }
constexpr uint64_t kAll = 1ull << 32, kChunk = 1 << 16;
template <typename F> static uint64_t over(uint64_t first, uint64_t last, uint64_t step, F differs) {
  uint64_t n = 0;
#pragma omp parallel for reduction(+ : n) schedule(static)
  for (uint64_t c = first; c < last; c += kChunk * step) {
    uint32_t k = 0;
    for (uint32_t i = 0; i < kChunk; ++i) k += differs(as_float((uint32_t)(c + i * step)));
    n += k;
  }
  return n;
}
// x / 15 and x / 9, finite x but -0 (see minus_zero)
extern "C" uint64_t division() {
  return over(0, kAll, 1, [](float x) -> uint32_t {
    const uint32_t wrong = (bits(dm_div15(x)) ^ bits(x / 15.0f)) | (bits(dm_div9(x)) ^ bits(x / 9.0f));
    return (wrong != 0u) & ((bits(x) & 0x7F800000u) != 0x7F800000u) & (bits(x) != 0x80000000u);
  });
}
extern "C" int minus_zero() { return dm_div15(-0.0f) == 0.0f && dm_div9(-0.0f) == 0.0f; }
// floor(x / 5) clamped to [0, 20], 9 - ceil(x / 5) clamped to [0, 8]; NaN: 0
static inline int clamp_class(float v, float top) {
  v = v < 0.0f ? 0.0f : (v > top ? top : v);
  return v != v ? 0 : (int)v;
}
extern "C" uint64_t classes() {
  return over(0, kAll, 1, [](float x) -> uint32_t {
    return (clamp_class(floorf(x * 0.2f), 20.0f) != clamp_class(floorf(x / 5.0f), 20.0f)) |
           (clamp_class(9.0f - ceilf(x * 0.2f), 8.0f) != clamp_class(9.0f - ceilf(x / 5.0f), 8.0f));
  });
}
// the exposure row from an aspect and a slope in degrees (lib.rs:472-614)
static inline float degrees(float rad) { return rad * 180.0f / 3.14159274101257324f; }
static inline int exposure(float sdeg, float adeg) {
  const float o = sdeg == 0.0f ? 180.0f : adeg;
  const int steep = sdeg <= 30.0f ? 0 : 1;
  if ((o >= 315.0f && o <= 360.0f) || (o >= 0.0f && o < 45.0f)) return steep;
  if (o >= 45.0f && o < 135.0f) return 2 + steep;
  if (o >= 135.0f && o < 225.0f) return 4 + steep;
  if (o >= 225.0f && o < 315.0f) return 6 + steep;
  return -1;
}
extern "C" uint64_t aspects(float slope) {
  const float sdeg = degrees(dm_atan_pos(slope));
  return over(0, kAll, 1, [=](float x) -> uint32_t { return dm_exposure(slope, x) != exposure(sdeg, degrees(x)); });
}
extern "C" uint64_t slopes(uint32_t first, uint64_t last, uint64_t step) {
  return over(first, last, step, [](float x) -> uint32_t { return dm_exposure(x, 1.0f) != exposure(degrees(dm_atan_pos(x)), degrees(1.0f)); });
}
"""


@pytest.fixture(scope="module")
def exhaustive(tmp_path_factory):
    d = tmp_path_factory.mktemp("dmoist_all")
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "e.cpp").write_text(EXHAUSTIVE)
    so = d / "e.so"
    subprocess.run(["g++", "-O3", "-std=c++17", "-march=x86-64-v3", "-fopenmp", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + str(d), "-I" + CSRC, str(d / "e.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    for f in ("division", "classes", "aspects", "slopes"):
        getattr(lib, f).restype = C.c_uint64
    lib.aspects.argtypes = [C.c_float]
    lib.slopes.argtypes = [C.c_uint32, C.c_uint64, C.c_uint64]
    return lib


def test_division_by_constants_for_every_finite_float(exhaustive):
    """-0 alone gives +0 (a difference of the interpolation's ends below 0.001 is
    not divided)."""
    assert exhaustive.division() == 0
    assert exhaustive.minus_zero()


def test_humidity_and_temperature_classes_for_every_float(exhaustive):
    assert exhaustive.classes() == 0


def test_exposure_limits(exhaustive):
    """The azimuths for every float, the slope of 30 degrees for every float from
    0.5 to 1 and every 31st of all."""
    assert exhaustive.aspects(0.4) == 0
    bits = lambda v: int(np.float32(v).view(np.uint32))  # noqa: E731
    assert exhaustive.slopes(bits(0.5), bits(1.0), 1) == 0
    assert exhaustive.slopes(0, 1 << 32, 31) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("month", [0, 13, -1, 12])
def test_months_on_the_device(pp, oracle, month):
    n = 5003
    x = _inputs(n, 7 + month)
    got = pp.dead_fuel_moisture(hour=14, month=month, **x)
    want = oracle.dmoist_cells(14, month, *[x[k] for k in x])
    for k, w in zip(("d1hr", "d10hr", "d100hr"), want):
        assert np.array_equal(got[k].view(np.uint32), w.view(np.uint32)), k
