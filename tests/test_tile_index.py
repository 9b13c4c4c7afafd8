"""Shared-memory tiles' index arithmetic (csrc/tile_index.cuh) on the host: the
slots of a launch's first sweep are the tile's own cells, each in exactly one
CTA's list, for every tile of up to 70 x 70 cells on every cluster size and for
long and wide ones, a single column or row among them; and the division is
exact over its range."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <vector>
#include "tile_index.cuh"
using namespace propag;
// 0, or the first thing wrong with a tile of TW x TH cells on C CTAs
extern "C" int tile(int TW, int TH, int C) {
  const int P = TW + 2, HR = TH + 2;
  std::vector<int> seen((size_t)P * HR, 0);
  for (int rank = 0; rank < C; ++rank)
    for (int k = 0; k < own_rows(TH, rank, C) * TW; ++k) {
      const int s = own_slot(k, rank, P, recip_of((uint32_t)TW));
      const int lr = (int)div_wide((uint32_t)s, recip_of((uint32_t)P));
      if (lr != s / P) return 1;
      const int hx = s - lr * P, hy = rank + lr * C;
      if (hx < 1 || hx > TW || hy < 1 || hy > TH) return 2;
      ++seen[(size_t)hy * P + hx];
    }
  for (int hy = 1; hy <= TH; ++hy)
    for (int hx = 1; hx <= TW; ++hx)
      if (seen[(size_t)hy * P + hx] != 1) return 3;
  return 0;
}
extern "C" int division(int d) {
  for (uint32_t s = 0; s < 65536; ++s)
    if (div_any(s, recip_of((uint32_t)d)) != s / (uint32_t)d) return 1;
  return 0;
}
"""


@pytest.fixture(scope="module")
def index(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    (d / "i.cpp").write_text(SOURCE)
    so = d / "i.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "propag-hidalgo_b200", "csrc"), str(d / "i.cpp"), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("ctas", [1, 2, 4, 8, 16])
def test_first_sweep_lists_every_cell_once(index, ctas):
    sizes = [(w, h) for w in range(1, 71) for h in range(1, 71)]
    sizes += [(1, 508), (508, 1), (2, 508), (323, 323), (1, 323), (508, 508 if ctas > 4 else 100)]
    for w, h in sizes:
        assert index.tile(w, h, ctas) == 0, (w, h)


def test_division_is_exact(index):
    for d in list(range(1, 700)) + [1023, 1024, 1025, 4095]:
        assert index.division(d) == 0, d
