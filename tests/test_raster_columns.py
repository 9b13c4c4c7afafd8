"""Polygon rows over the polygon's own columns (csrc/raster_kernels.cuh), at the
forms where the columns could be cut wrongly: polygons left and right of the
grid and across its edges, vertices far away, infinite and NaN vertices, on
grids with eight threads, a warp and a CTA to a row (up to 4096, up to 16384, more).  The emulated
kernels' rasters equal the host rasteriser's, which looks at every column."""
import ctypes as C

import numpy as np
import pytest

from test_raster import georef, wkb_polygon
from test_raster_kernels_emulated import L, _features, _host_fuels, emul  # noqa: F401 (fixtures)


def _rings(w, h, rng):
    def box(x0, y0, x1, y1):
        return [(x0, y0), (x1, y0), (x1, y1), (x0, y1), (x0, y0)]
    rings = [box(-9.0, 0.5, -2.0, h - 0.5), box(w + 2.0, 0.2, w + 9.0, h - 0.2),       # beside the grid
             box(-5.0, 0.4, 3.5, 2.6), box(w - 2.5, 0.6, w + 4.0, h + 3.0),              # across an edge
             box(31.5, 0.0, 32.5, h), box(31.49, 1.0, 64.51, 2.0),                       # mask word edges
             [(-1e12, 1.0), (1e12, 1.5), (0.5 * w, 3.0), (-1e12, 1.0)],                  # far away
             [(5.0, 0.0), (np.inf, 2.0), (9.0, 4.0), (5.0, 0.0)],
             [(5.0, 0.0), (np.nan, 2.0), (9.0, 4.0), (5.0, 0.0)],
             [(0.3 * w, -1e300), (0.6 * w, 1e300), (0.1 * w, 2.0), (0.3 * w, -1e300)]]
    for _ in range(12):
        n = int(rng.integers(3, 9))
        xs, ys = rng.uniform(-0.2 * w, 1.2 * w, n), rng.uniform(-2, h + 2, n)
        rings.append([(float(x), float(y)) for x, y in zip(xs, ys)])
        rings[-1].append(rings[-1][0])
    return rings


@pytest.mark.parametrize("w", [70, 4096, 4097, 8192, 8193, 16384, 16385])
def test_polygon_columns(L, emul, w):  # noqa: F811
    h = 5
    g = georef(L, w, h, (0.0, 1.0, 0.0, 0.0, 0.0, 1.0))
    rings = _rings(w, h, np.random.default_rng(w))
    for order in (rings, rings[::-1]):
        items = [(k, wkb_polygon([r])) for k, r in enumerate(order)]
        arr, keep = _features(L, L.FFIFuelFeature, items, "code")
        expect = _host_fuels(L, g, arr, len(items))
        got = np.empty(w * h, np.uint8)
        emul.emul_rasterize_fuels(C.addressof(arr), len(items), C.addressof(g), got.ctypes.data, 3)
        assert np.array_equal(got, expect)
        assert np.count_nonzero(expect != 255) > 20
