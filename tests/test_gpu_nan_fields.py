"""Fire fields with NaN (from terrain without data) and infinite speeds: a
neighbour whose offer is NaN is passed over, as in the reference's loop of
comparisons (crates/propag/src/propag.cu:124-190), and hides no other
neighbour's.  Times, references and counters equal the oracle's (exact
comparison: the same operations on the same values)."""
import numpy as np
import pytest

from conftest import trig_for
from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _job

pytestmark = pytest.mark.gpu


# global-memory tiles, shared-memory tiles, several teams
@pytest.mark.parametrize("size,tile,cluster", [(150, 64, 0), (150, 64, 4), (150, -1, 16), (450, 86, -20), (700, 86, 0)])
@pytest.mark.parametrize("arith", [0, 1])
def test_nan_fields(pp, ref_oracle, size, tile, cluster, arith):
    import torch
    from py_propag import _lib as L
    from py_propag import scenarios as S
    sc = S.config1(size=size, seed=48, n_ign=4, max_time=15000.0)
    d = _device_scenario(pp, sc)
    rng = np.random.default_rng(size + cluster)
    fields = {k: d[k].cpu().numpy() for k in ("sp", "az", "ec")}
    for k, values in (("sp", [np.nan, np.nan, np.inf]), ("az", [np.nan]), ("ec", [np.nan, 0.0, 1.0])):
        at = rng.random(size * size) < 0.015
        fields[k][at] = rng.choice(np.array(values, np.float32), int(at.sum()))
        d[k].copy_(torch.from_numpy(fields[k]))
    eng = pp.Engine(cluster=cluster)
    st = eng.run([_job(L, size, size, sc.dx, sc.dy, sc.max_time, d, tile=tile, arith=arith)])[0]
    torch.cuda.synchronize()
    eng.close()
    o = ref_oracle.propagate(size, size, sc.dx, sc.dy, sc.max_time, *[fields[k] for k in ("sp", "az", "ec")],
                             sc.ignitions, tile=(0 if tile == -1 else tile), full=(0 if cluster > 0 else 2),
                             trig=trig_for(arith))
    time = d["time"].cpu().numpy()
    assert np.array_equal(time.view(np.uint32), o.time.ravel().view(np.uint32))
    assert np.array_equal(d["rx"].cpu().numpy().view(np.uint16), o.refs_x.ravel())
    assert np.array_equal(d["ry"].cpu().numpy().view(np.uint16), o.refs_y.ravel())
    for k in SCHEDULE + WORK:
        assert st[k] == o.stats[k], k
    assert st["burned"] > 500
