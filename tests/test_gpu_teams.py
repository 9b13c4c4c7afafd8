"""Global-memory tiles at the edges of their bookkeeping: work lists taken in
several chunks, update entries beyond shared memory, tiles whose last group of
cells is ragged, walks beyond the closed form and referrer boxes scanned by
the whole CTA.  Times, references and schedule counters equal the oracle's
(exact comparison: the same operations in the same order)."""
import numpy as np
import pytest

from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _job

pytestmark = pytest.mark.gpu


def _uniform(pp, n, max_time):
    """Constant ground: one ignition is every cell's reference, so walks and
    referrer boxes grow with the fire."""
    from py_propag import scenarios as S
    return S.Scenario(n, n, 5.0, 5.0, max_time, pp.demo_terrain(n, n), [(3, n - 2, 0.0), (n // 2, n // 3, 900.0)])


# (threads, jobs, team size): 50 jobs of a device with at least 148 resident
# CTAs leave teams of a few CTAs; 32 threads make 1 024-entry lists and
# one-warp CTAs
@pytest.mark.parametrize("threads,copies,cluster", [(512, 17, -2), (32, 17, -2), (96, 1, -7), (512, 1, 0)])
def test_teams_and_chunks(pp, ref_oracle, threads, copies, cluster):
    import torch
    from py_propag import _lib as L
    from py_propag import scenarios as S
    scs = [S.config1(size=150, seed=31, n_ign=700, max_time=3000.0),  # many updates in the first sweeps
           S.config1(size=131, seed=32, n_ign=5, max_time=9000.0),    # 17 161 cells: a group of one
           _uniform(pp, 190, 30000.0)]                                # offsets past the closed form's 127
    devs = [[_device_scenario(pp, sc) for sc in scs] for _ in range(copies)]
    jobs = [_job(L, sc.width, sc.height, sc.dx, sc.dy, sc.max_time, d, tile=(-1 if i != 1 else 53))
            for row in devs for i, (sc, d) in enumerate(zip(scs, row))]
    eng = pp.Engine(cluster=cluster, threads=threads)
    stats = eng.run(jobs)
    torch.cuda.synchronize()
    eng.close()
    for i, sc in enumerate(scs):
        sp, az, ec = (devs[0][i][k].cpu().numpy() for k in ("sp", "az", "ec"))
        o = ref_oracle.propagate(sc.width, sc.height, sc.dx, sc.dy, sc.max_time, sp, az, ec, sc.ignitions,
                                 tile=(0 if i != 1 else 53), full=2, trig=3)
        for row in range(copies):
            d, st = devs[row][i], stats[3 * row + i]
            assert np.array_equal(d["time"].cpu().numpy().view(np.uint32), o.time.ravel().view(np.uint32)), (i, row)
            assert np.array_equal(d["rx"].cpu().numpy().view(np.uint16), o.refs_x.ravel()), (i, row)
            assert np.array_equal(d["ry"].cpu().numpy().view(np.uint16), o.refs_y.ravel()), (i, row)
            for k in SCHEDULE + WORK:
                assert st[k] == o.stats[k], (i, row, k)
    assert max(s["max_walk"] for s in stats) > 127
