"""Shared-memory tiles whose updates some warps commit while the others walk
their lines of sight (csrc/engine.cu, tile_smem): CTAs of one warp, which does
both, of two and three, and whole ones, with more updates in a sweep than the
walking warps hold and walks past the closed form.  Times, references and
schedule counters equal the oracle's (exact comparison: the same operations in
the same order)."""
import numpy as np
import pytest

from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _job
from test_gpu_teams import _uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,cluster", [(32, 4), (64, 2), (96, 4), (512, 1), (512, 8)])
def test_commit_and_walk_warps(pp, ref_oracle, threads, cluster):
    import torch
    from py_propag import _lib as L
    from py_propag import scenarios as S
    scs = [S.config1(size=110, seed=41, n_ign=400, max_time=3000.0),
           S.config1(size=97, seed=42, n_ign=3, max_time=9000.0),
           _uniform(pp, 150, 30000.0)]
    tiles = (64, 53, 150)
    devs = [_device_scenario(pp, sc) for sc in scs]
    jobs = [_job(L, sc.width, sc.height, sc.dx, sc.dy, sc.max_time, d, tile=t) for sc, d, t in zip(scs, devs, tiles)]
    eng = pp.Engine(cluster=cluster, threads=threads)
    stats = eng.run(jobs)
    torch.cuda.synchronize()
    eng.close()
    for i, sc in enumerate(scs):
        sp, az, ec = (devs[i][k].cpu().numpy() for k in ("sp", "az", "ec"))
        d, st = devs[i], stats[i]
        # 152 x 152 staged cells of 12 bytes do not fit one CTA: that tile stays in
        # global memory, whose first sweeps evaluate the pending cells only
        full = 2 if cluster == 1 and tiles[i] == 150 else 0
        o = ref_oracle.propagate(sc.width, sc.height, sc.dx, sc.dy, sc.max_time, sp, az, ec, sc.ignitions,
                                 tile=tiles[i], full=full, trig=3)
        assert np.array_equal(d["time"].cpu().numpy().view(np.uint32), o.time.ravel().view(np.uint32)), i
        assert np.array_equal(d["rx"].cpu().numpy().view(np.uint16), o.refs_x.ravel()), i
        assert np.array_equal(d["ry"].cpu().numpy().view(np.uint16), o.refs_y.ravel()), i
        for k in SCHEDULE + WORK:
            assert st[k] == o.stats[k], (i, k)
    assert max(s["max_walk"] for s in stats) > 127
