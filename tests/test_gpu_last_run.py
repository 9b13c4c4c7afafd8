"""What the engine says about how its last run was launched, at the sizes where
several teams begin to share a lone job."""
import ctypes as C

import pytest

from test_gpu_propag import _device_scenario, _job

pytestmark = pytest.mark.gpu


# windows of one, two and three tiles: four, six and eight tiles along a side
@pytest.mark.parametrize("size,tile,jobs,cluster,shared", [
    (772, 257, 1, 0, True), (771, 257, 1, 0, False), (751, 150, 1, 0, True), (750, 150, 1, 0, False),
    (603, 86, 1, 0, True), (602, 86, 1, 0, False), (772, 257, 2, 0, False), (772, 257, 1, -148, False),
    (772, 257, 1, 8, False), (700, 85, 1, 0, False)])
def test_last_run(pp, size, tile, jobs, cluster, shared):
    from py_propag import _lib as L
    from py_propag import scenarios as S
    sc = S.Scenario(size, size, 5.0, 5.0, 200.0, pp.demo_terrain(size, size), [(size // 2, size // 2, 0.0)])
    devs = [_device_scenario(pp, sc) for _ in range(jobs)]
    eng = pp.Engine(cluster=cluster)
    kernels, teams = C.c_uint32(), C.c_uint32()
    ask = lambda: L.lib().propag_engine_last_run(eng._h, C.byref(kernels), C.byref(teams))  # noqa: E731
    assert ask() == L.PROPAG_ERR_INVALID  # nothing has run
    eng.run([_job(L, size, size, sc.dx, sc.dy, sc.max_time, d, tile=tile) for d in devs])
    assert ask() == 0
    assert (kernels.value, teams.value > 0) == ((8, True) if shared else (4, False))
    eng.close()
