"""How often the fire pass's moisture sums (csrc/moist_sums.cuh) fall back from
double to double-float, on the host: rarely on ordinary moistures -- the double
sums are what the pass runs -- and often where sums lie on ties between two
floats, so that both ways are among what the bit comparisons compare."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_moist_sums import _moistures

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "propag-hidalgo_b200", "csrc")

SOURCE = r"""
#include "moist_sums.cuh"
using namespace propag;
static FuelConst table[kMaxFuels];
// cells whose double sums are not trusted
extern "C" long moist_fallbacks(long n, const int *fuel, const float *m) {
  if (!build_catalog_table(table)) return -1;
  long k = 0;
  for (long i = 0; i < n; ++i) {
    Moist r;
    k += !moist_double(table[fuel[i]], m + 5 * i, r);
  }
  return k;
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
    lib.moist_fallbacks.restype = C.c_long
    return lib


def _share(sums, kind, fuel=None):
    n = 400_000
    rng = np.random.default_rng(len(kind))
    m = _moistures(kind, n, rng)
    fuel = (rng.integers(1, 14, n) if fuel is None else np.full(n, fuel)).astype(np.int32)
    k = sums.moist_fallbacks(C.c_long(n), fuel.ctypes.data_as(C.c_void_p), m.ctypes.data_as(C.c_void_p))
    assert k >= 0
    return k / n


def test_ordinary_moistures_run_in_double(sums):
    assert _share(sums, "ordinary") < 0.01
    for f in range(1, 14):
        assert _share(sums, "ordinary", f) < 0.01, f


@pytest.mark.parametrize("kind", ["percent grid", "extinction", "wide"])
def test_ties_and_extremes_fall_back(sums, kind):
    assert 0.0 < _share(sums, kind) < 1.0
