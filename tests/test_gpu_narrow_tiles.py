"""Shared-memory tiles one cell wide: grids of one column, and grids whose last
tile column is one cell wide (width % tile == 1), on explicit clusters with both
referrer-box codecs and through the allocation-free entry point.  The fire
starts on the left, so the last column burns from its left neighbour.  Times,
references and schedule and work counters equal the oracle's (exact comparison:
the same operations in the same order)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _job

pytestmark = pytest.mark.gpu


def _scenario(width, height):
    from py_propag import scenarios as S
    sc = S.config1(size=400, seed=44, n_ign=1, max_time=20000.0)
    terrain = {k: np.ascontiguousarray(v[:height, :width]) for k, v in sc.terrain.items()}
    fuel = terrain["fuel_code"]
    burnable = [(x, y) for x in range(max(width // 2, 1)) for y in range(height) if fuel[y, x]]
    ign = [(*burnable[i * len(burnable) // 3], 200.0 * i) for i in range(3)]
    # the last column and the one before it burn along their whole length
    fuel[:, max(width - 2, 0):] = 1
    return S.Scenario(width, height, 5.0, 5.0, sc.max_time, terrain, ign)


def _compare(ref_oracle, sc, d, st, tile):
    sp, az, ec = (d[k].cpu().numpy() for k in ("sp", "az", "ec"))
    o = ref_oracle.propagate(sc.width, sc.height, sc.dx, sc.dy, sc.max_time, sp, az, ec, sc.ignitions,
                             tile=(0 if tile == -1 else tile or 323), full=0, trig=3)
    time = d["time"].cpu().numpy().reshape(sc.height, sc.width)
    assert np.array_equal(time.view(np.uint32), o.time.view(np.uint32))
    assert np.array_equal(d["rx"].cpu().numpy().view(np.uint16), o.refs_x.ravel())
    assert np.array_equal(d["ry"].cpu().numpy().view(np.uint16), o.refs_y.ravel())
    for k in SCHEDULE + WORK:
        assert st[k] == o.stats[k], k
    assert np.mean(time[:, -1] < np.finfo(np.float32).max) > 0.3


# 16 bytes a staged cell fit 16 CTAs at a tile of 323 (exact referrer boxes) and
# not eight (coarse ones)
@pytest.mark.parametrize("width,height,tile,cluster", [
    (1, 37, -1, 1), (1, 300, -1, 4), (1, 300, 64, 16), (129, 90, 64, 2), (129, 140, 128, 4), (257, 60, 128, 16),
    (324, 200, 323, 16), (324, 330, 323, 8), (65, 65, 64, 1), (60, 129, 64, 8), (2, 70, 1, 2)])
def test_one_cell_wide(pp, ref_oracle, width, height, tile, cluster):
    import torch
    from py_propag import _lib as L
    sc = _scenario(width, height)
    d = _device_scenario(pp, sc)
    eng = pp.Engine(cluster=cluster)
    st = eng.run([_job(L, width, height, sc.dx, sc.dy, sc.max_time, d, tile=tile)])[0]
    torch.cuda.synchronize()
    eng.close()
    _compare(ref_oracle, sc, d, st, tile)


@pytest.mark.parametrize("width,height,tile", [(1, 200, 0), (129, 90, 64), (324, 200, 0)])
def test_one_cell_wide_allocation_free(pp, ref_oracle, width, height, tile):
    import torch
    from py_propag import _lib as L
    sc = _scenario(width, height)
    d = _device_scenario(pp, sc)
    job = _job(L, width, height, sc.dx, sc.dy, sc.max_time, d, tile=tile)
    st = L.PropagStats()
    assert L.lib().propag_run_device_static(C.byref(job), None, C.byref(st)) == 0, L.last_error()
    torch.cuda.synchronize()
    _compare(ref_oracle, sc, d, st.as_dict(), tile)
