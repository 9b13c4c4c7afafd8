"""The closed form of the line-of-sight walk (csrc/dda_columns.cuh) against
the step-by-step walk of the reference (crates/propag/src/propag.h:91-135, the
oracle's restatement): the same cells in the same order for every offset it
covers, in every direction's axis order, and the count of visited cells."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "dda_columns.cuh"
using namespace propag;
static float table[kCrossTableLen];
extern "C" int columns_max() { return kColumnsMax; }
extern "C" void columns_init() {
  for (int n = 1; n <= kColumnsMax; ++n) {
    const float step = 1.0f / (float)n;
    float t = step;
    for (int i = 1; i <= n; ++i, t += step) table[cross_at(n, i)] = t;
  }
}
// Cells (column, row) of the walk in order, their order index c + r - diagonal
// steps, and the visited count P + Q + 1 - diagonal steps.
extern "C" int columns_walk(int P, int Q, int *cells, int *order, int *visited) {
  int k = 0, diags = 0;
  for (int c = 0; c <= P; ++c) {
    int jin, jout;
    bool diag;
    walk_column(table, P, Q, c, 1.0f / (float)P, jin, jout, diag);
    diags += diag;
    if (jout < jin || jout > jin + 1) return -1;
    for (int r = jin; r <= jout; ++r, ++k) {
      cells[2 * k] = c;
      cells[2 * k + 1] = r;
      order[k] = c + r - diags;
    }
  }
  *visited = P + Q + 1 - diags;
  return k;
}
"""


@pytest.fixture(scope="module")
def columns(tmp_path_factory):
    d = tmp_path_factory.mktemp("columns")
    (d / "columns.cpp").write_text(SOURCE)
    so = d / "columns.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "propag-hidalgo_b200", "csrc"), str(d / "columns.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    lib.columns_init()
    return lib


@pytest.mark.parametrize("swap", [False, True])
def test_every_covered_offset(columns, oracle, swap):
    lib = oracle._load()
    lib.ops_dda_cells.restype = C.c_int64
    n = columns.columns_max()
    room = 4 * n + 8
    cells, order = (np.zeros(2 * room, np.int32), np.zeros(room, np.int32))
    walk = np.zeros(2 * room, np.int32)
    visited = C.c_int(0)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    for P in range(1, n + 1):
        for Q in range(0, P + 1):
            k = columns.columns_walk(P, Q, ptr(cells), ptr(order), C.byref(visited))
            tx, ty = (Q, P) if swap else (P, Q)
            m = lib.ops_dda_cells(0, 0, tx, ty, ptr(walk), C.c_int64(room))
            assert k == m == visited.value, (P, Q)
            got = cells[:2 * k].reshape(-1, 2)
            want = walk[:2 * k].reshape(-1, 2)
            if swap:
                want = want[:, ::-1]
            assert np.array_equal(got, want), (P, Q)
            assert np.array_equal(order[:k], np.arange(k)), (P, Q)
