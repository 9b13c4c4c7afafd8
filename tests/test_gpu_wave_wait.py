"""The bounded waits of several teams on one job (csrc/engine.cu, waves_kernel):
a tile that no team may take makes every wait run out; the run fails with the
timeout status, is not repeated in sequence, and the next run on the same engine
equals the oracle (exact comparison)."""
import ctypes as C
import time

import numpy as np
import pytest

from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _job

pytestmark = pytest.mark.gpu


def _run(L, job, hold, limit_ms):
    st = (L.PropagStats * 2)()
    t0 = time.perf_counter()
    rc = L.lib().propag_selftest_wave_wait(C.byref(job), hold, limit_ms, st)
    return rc, time.perf_counter() - t0, st[0].as_dict(), st[1].as_dict()


def _equals_oracle(ref_oracle, sc, d, st, tile):
    sp, az, ec = (d[k].cpu().numpy() for k in ("sp", "az", "ec"))
    o = ref_oracle.propagate(sc.width, sc.height, sc.dx, sc.dy, sc.max_time, sp, az, ec, sc.ignitions, tile=tile,
                             full=2, trig=3)
    assert np.array_equal(d["time"].cpu().numpy().view(np.uint32), o.time.ravel().view(np.uint32))
    assert np.array_equal(d["rx"].cpu().numpy().view(np.uint16), o.refs_x.ravel())
    assert np.array_equal(d["ry"].cpu().numpy().view(np.uint16), o.refs_y.ravel())
    for k in SCHEDULE + WORK:
        assert st[k] == o.stats[k], k


# windows of one, two and three tiles
@pytest.mark.parametrize("size,tile", [(1100, 257), (1100, 150), (760, 86)])
def test_teams_give_up_and_the_engine_stays_usable(pp, ref_oracle, size, tile):
    from py_propag import _lib as L
    from py_propag import scenarios as S
    sc = S.config1(size=size, seed=46, n_ign=5, max_time=9000.0)
    d = _device_scenario(pp, sc)
    job = _job(L, size, size, sc.dx, sc.dy, sc.max_time, d, tile=tile)
    # the tile of the first ignition: what lies around it waits for it
    x, y, _ = sc.ignitions[0]
    hold = x // tile + (y // tile) * -(-size // tile)
    rc, seconds, first, second = _run(L, job, hold, 40)
    assert rc == L.PROPAG_ERR_TIMEOUT, L.last_error()
    assert "gave up" in L.last_error()
    assert first["status"] == 2 and second["status"] == 0
    assert seconds < 10.0
    # not repeated: a run in sequence makes every improvement
    assert first["improvements"] < second["improvements"]
    _equals_oracle(ref_oracle, sc, d, second, tile)


def test_jobs_without_teams_and_tiles_outside_are_refused(pp):
    from py_propag import _lib as L
    from py_propag import scenarios as S
    sc = S.config1(size=150, seed=46, n_ign=2, max_time=3000.0)
    d = _device_scenario(pp, sc)
    small = _job(L, 150, 150, sc.dx, sc.dy, sc.max_time, d, tile=0)
    assert _run(L, small, -1, 40)[0] == L.PROPAG_ERR_INVALID
    assert _run(L, small, 1, 40)[0] == L.PROPAG_ERR_INVALID


def test_long_launches_are_not_taken_for_a_stall(pp):
    """A team waits for another one's launch as long as that one goes on: launches
    that take many times the limit, a sweep every few microseconds."""
    from py_propag import _lib as L
    from py_propag import scenarios as S
    size, tile = 1640, 410
    sc = S.Scenario(size, size, 5.0, 5.0, 1.0e4, pp.demo_terrain(size, size), [(615, 615, 0.0)])
    d = _device_scenario(pp, sc)
    job = _job(L, size, size, sc.dx, sc.dy, sc.max_time, d, tile=tile)
    rc, _, first, second = _run(L, job, -1, 2)
    assert rc == 0, L.last_error()
    assert first["status"] == second["status"] == 0 and first["burned"] > 20000
    for k in SCHEDULE + WORK:
        assert first[k] == second[k], k
