"""The fire pass's moisture sums (csrc/moist_sums.cuh) on the CPU: the double
sums with their check give the double-float sums' floats bit for bit, on
ordinary moistures, near and past the moisture of extinction, at ties between
two floats, on wide ranges and on negative, infinite and NaN inputs; and the
check rarely calls for the double-float sums on ordinary moistures."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "propag-hidalgo_b200", "csrc")

SOURCE = r"""
#include "moist_sums.cuh"
using namespace propag;
static FuelConst table[kMaxFuels];
extern "C" int moist_init() { return build_catalog_table(table) ? 0 : -1; }
extern "C" void moist_run(long n, const int *fuel, const float *m, float *both) {
  for (long i = 0; i < n; ++i) {
    const FuelConst &F = table[fuel[i]];
    const float *v = m + 5 * i;
    const Moist a = moist_sums(F, v), b = moist_df(F, v[0], v[1], v[2], v[3], v[4]);
    const float r[6] = {a.dead, a.live, a.lmext, b.dead, b.live, b.lmext};
    for (int k = 0; k < 6; ++k) both[6 * i + k] = r[k];
  }
}
"""


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    d = tmp_path_factory.mktemp("moist")
    (d / "m.cpp").write_text(SOURCE)
    so = d / "m.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-shared", "-fPIC", "-I" + CSRC,
                    str(d / "m.cpp"), os.path.join(CSRC, "catalog.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    assert lib.moist_init() == 0
    return lib


def _moistures(kind, n, rng):
    if kind == "ordinary":
        m = np.array([0.06, 0.07, 0.08, 0.6, 0.9]) + rng.uniform(-0.02, 0.02, (n, 5))
    elif kind == "percent grid":  # many ties: multiples of 1/100 and 1/256
        m = np.where(rng.random((n, 5)) < 0.5, rng.integers(0, 101, (n, 5)) / 100, rng.integers(0, 257, (n, 5)) / 256)
    elif kind == "extinction":
        m = np.repeat(rng.choice([0.12, 0.15, 0.2, 0.25, 0.3, 0.4], (n, 1)), 5, 1) * (1 + rng.normal(0, 1e-6, (n, 5)))
        m[:, 3:] = rng.uniform(0.3, 3.0, (n, 2))
    else:
        m = rng.uniform(0, 1, (n, 5)) * 10.0 ** rng.uniform(-6, 4, (n, 5))
        for v in (0.0, np.inf, -np.inf, np.nan):
            m[rng.random((n, 5)) < 0.01] = v
        m[rng.random((n, 5)) < 0.03] *= -1
    return np.ascontiguousarray(m, np.float32)


@pytest.mark.parametrize("kind", ["ordinary", "percent grid", "extinction", "wide"])
def test_double_sums_round_as_double_float(sums, kind):
    n = 400_000
    rng = np.random.default_rng(len(kind))
    m = _moistures(kind, n, rng)
    fuel = rng.integers(1, 14, n).astype(np.int32)
    both = np.zeros((n, 6), np.float32)
    sums.moist_run(C.c_long(n), fuel.ctypes.data_as(C.c_void_p), m.ctypes.data_as(C.c_void_p),
                   both.ctypes.data_as(C.c_void_p))
    a, b = both[:, :3], both[:, 3:]
    # a numerator that is not positive counts as zero whatever its value, and
    # the live numbers of a model without live fuel are not read
    live = np.isin(fuel, (2, 4, 5, 7, 10))
    for k, used in ((0, np.ones(n, bool)), (1, live), (2, live)):
        p, q = a[used, k], b[used, k]
        if k < 2:
            p, q = np.where(p > 0, p, 0), np.where(q > 0, q, 0)
            assert np.array_equal(p.view(np.uint32), q.view(np.uint32)), k
        else:  # the denominator is read where the live numerator is positive
            on = np.where(b[used, 1] > 0, True, False)
            assert np.array_equal(p[on].view(np.uint32), q[on].view(np.uint32)), k
