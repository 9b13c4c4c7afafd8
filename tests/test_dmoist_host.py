"""The dmoist model's device code (csrc/dmoist_device.cuh) compiled for the
host, against the CPU restatement of the reference (crates/dmoist/src/
lib.rs:55-715): equal bit for bit in every month a caller can pass, the ones
outside 1..12 included, for which the reference has no shading correction (the
corrected humidity class is NaN there, and every moisture zero)."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("month", [0, 13, -1, 12])
def test_months_on_the_device(pp, oracle, month):
    n = 5003
    x = _inputs(n, 7 + month)
    got = pp.dead_fuel_moisture(hour=14, month=month, **x)
    want = oracle.dmoist_cells(14, month, *[x[k] for k in x])
    for k, w in zip(("d1hr", "d10hr", "d100hr"), want):
        assert np.array_equal(got[k].view(np.uint32), w.view(np.uint32)), k
