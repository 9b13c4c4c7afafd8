"""Several teams on one job: launches of independent tiles at the same time
give the sequence's results.  Times, references and every schedule and work
counter equal the oracle's, which runs the launches one after another (exact
comparison: the same operations on the same values)."""
import numpy as np
import pytest

from conftest import trig_for
from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _fire, _job, _settings

pytestmark = pytest.mark.gpu


def _scenario(pp, kind, size):
    from py_propag import scenarios as S
    if kind == "ridges":
        return S.config1(size=size, seed=41, n_ign=9, max_time=20000.0)
    if kind == "one":
        return S.config1(size=size, seed=42, n_ign=1, max_time=30000.0)
    # constant ground: references further away than the window allows, so the
    # job is started again in sequence
    return S.Scenario(size, size, 5.0, 5.0, 6.0e4, pp.demo_terrain(size, size),
                      [(size // 2, size // 3, 0.0), (10, size - 20, 3000.0)])


# tiles of 257 cells or more: a window of one tile; 129 to 256: two; 86 to 128: three
@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("kind,size,tile", [("ridges", 1100, 257), ("ridges", 1100, 150), ("ridges", 760, 86),
                                            ("one", 1100, 257), ("constant", 800, 100)])
def test_waves_equal_the_sequence(pp, ref_oracle, kind, size, tile, arith):
    sc = _scenario(pp, kind, size)
    s = _settings(pp, sc.width, sc.height, sc.dx, sc.dy, sc.max_time)
    res = pp.propagate_arrays(s, sc.terrain, sc.ignitions, tile=tile, arith=arith)
    sp, az, ec = _fire(pp, sc.terrain)
    o = ref_oracle.propagate(sc.width, sc.height, sc.dx, sc.dy, sc.max_time, sp, az, ec, sc.ignitions, tile=tile,
                             full=2, trig=trig_for(arith))
    assert np.array_equal(res.arrival_times.view(np.uint32), o.time.view(np.uint32))
    assert np.array_equal(res.refs_x.reshape(sc.height, sc.width), o.refs_x)
    assert np.array_equal(res.refs_y.reshape(sc.height, sc.width), o.refs_y)
    for k in SCHEDULE + WORK:
        assert res.stats[k] == o.stats[k], k
    if kind == "constant":  # the longest line of sight spans more than three tiles
        assert res.stats["max_walk"] > 3 * tile


def test_waves_without_ignition_and_in_a_graph(pp):
    """No ignition: one round of empty launches.  As a CUDA graph, replayed: the
    same results each time."""
    import torch
    from py_propag import _lib as L
    from py_propag import scenarios as S
    sc = S.config1(size=1100, seed=43, n_ign=6, max_time=9000.0)
    for ignitions in ([], sc.ignitions):
        sc.ignitions = ignitions
        d = _device_scenario(pp, sc)
        job = _job(L, sc.width, sc.height, sc.dx, sc.dy, sc.max_time, d, tile=257)
        eng = pp.Engine()
        st = eng.run([job])[0]
        eng.close()
        times = d["time"].clone()
        assert (st["rounds"], st["sweeps"]) == (1, 25) if not ignitions else st["rounds"] > 1
        g = pp.Graph([job], None)
        for _ in range(2):
            d["time"].zero_()
            g.launch()
            torch.cuda.synchronize()
            assert torch.equal(d["time"].view(torch.int32), times.view(torch.int32))
            again = g.stats()[0]
            assert all(again[k] == st[k] for k in SCHEDULE + WORK)
        g.close()
