"""The device memory that the rasterisers keep between calls is given back when
the caller asks for it (propag_trim_scratch), and they work as before then."""
import ctypes as C

import numpy as np
import pytest

from test_raster import georef, wkb_polygon


def test_nothing_kept(pp):
    from py_propag import _lib as L
    assert L.lib().propag_trim_scratch() == L.PROPAG_OK


@pytest.mark.gpu
def test_kept_memory_is_given_back(pp):
    import torch
    from py_propag import _lib as L
    from test_zz_raster_device import _fuel_features
    lib = L.lib()
    w, h = 4000, 3500
    g = georef(L, w, h, (0.0, 4.0, 0.0, 0.0, 0.0, 4.0))
    ring = [(50.0, 50.0), (15000.0, 60.0), (14000.0, 13000.0), (70.0, 12000.0), (50.0, 50.0)]
    arr, keep = _fuel_features(L, [(3, wkb_polygon([ring]))])
    crs = bytes(g.proj).rstrip(b"\0")
    d = torch.zeros(w * h, dtype=torch.uint8, device="cuda")

    def run():
        assert lib.propag_rasterize_fuels_device(arr, 1, crs, C.byref(g), d.data_ptr(), None) == 0, L.last_error()
        torch.cuda.synchronize()
        return d.cpu().numpy().copy()

    first = run()
    assert (first == 3).mean() > 0.5 and (first == 255).any()
    assert lib.propag_trim_scratch() == 0
    free0 = torch.cuda.mem_get_info()[0]
    run()  # 56 MB of winners, below the 128 MiB that are kept
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert 4 * w * h <= kept <= (128 << 20) + (64 << 20)
    assert lib.propag_trim_scratch() == 0
    assert abs(torch.cuda.mem_get_info()[0] - free0) < 4 << 20
    assert np.array_equal(run(), first)
