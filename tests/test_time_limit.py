"""A job without a time limit (max_time infinite): a cell that has not burned,
whose time is FLT_MAX and which has no reference, never counts as burning, and
the results are those of the limit FLT_MAX."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FMAX = float(np.finfo(np.float32).max)


def test_no_unburned_cell_lies_below_the_limit(tmp_path):
    """The kernels' test (time < limit) for a cell that has not burned, and for
    the latest time that a burned cell can have, for every kind of limit."""
    (tmp_path / "t.cpp").write_text('#include "engine.cuh"\n'
                                    'extern "C" float limit(float m) { return propag::time_limit(m); }\n')
    so = tmp_path / "t.so"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(cuda, "include"),
                    "-I" + os.path.join(ROOT, "propag-hidalgo_b200", "csrc"), str(tmp_path / "t.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    lib.limit.argtypes, lib.limit.restype = [C.c_float], C.c_float
    latest = float(np.nextafter(np.float32(FMAX), np.float32(0)))
    for m in map(float, np.array([0.0, -1.0, 1e-40, 3600.0, latest, FMAX, np.inf, -np.inf, np.nan], np.float32)):
        t = lib.limit(m)
        assert not FMAX < t, m
        assert (latest < t) == (m >= FMAX), m
        if not m == np.inf:
            assert t == m or np.isnan(m) and np.isnan(t)


@pytest.mark.gpu
@pytest.mark.parametrize("cluster", [0, 4, "static", "host"])
@pytest.mark.parametrize("arith", [0, 1])
def test_infinite_limit(pp, ref_oracle, cluster, arith):
    import torch
    from conftest import trig_for
    from py_propag import _lib as L
    from py_propag import scenarios as S
    from test_gpu_propag import SCHEDULE, WORK, _device_scenario, _job
    sc = S.config1(size=150, seed=45, n_ign=4, max_time=1e30)
    d = _device_scenario(pp, sc)
    job = _job(L, 150, 150, sc.dx, sc.dy, np.inf, d, tile=64, arith=arith)
    if cluster == "static":
        st = L.PropagStats()
        assert L.lib().propag_run_device_static(C.byref(job), None, C.byref(st)) == 0, L.last_error()
        st = st.as_dict()
    elif cluster == "host":
        gt = [0.0, sc.dx, 0.0, 0.0, 0.0, sc.dy]
        settings = pp.PySettings(pp.PyGeoReference(150, 150, "+proj=utm +zone=30 +ellps=GRS80 +units=m +no_defs", gt),
                                 1000.0)
        settings._max_time = np.inf  # a C caller's limit: the class takes finite ones only
        res = pp.propagate_arrays(settings, sc.terrain, sc.ignitions, tile=64, arith=arith)
        st = res.stats
        for k, v in (("time", res.arrival_times), ("rx", res.refs_x), ("ry", res.refs_y)):
            d[k].copy_(torch.from_numpy(np.ascontiguousarray(v).view({2: np.int16, 4: np.float32}[v.itemsize]).ravel()))
    else:
        eng = pp.Engine(cluster=cluster)
        st = eng.run([job])[0]
        eng.close()
    torch.cuda.synchronize()
    sp, az, ec = (d[k].cpu().numpy() for k in ("sp", "az", "ec"))
    o = ref_oracle.propagate(150, 150, sc.dx, sc.dy, FMAX, sp, az, ec, sc.ignitions, tile=64,
                             full=(2 if cluster in (0, "host") else 0), trig=trig_for(arith))
    assert np.array_equal(d["time"].cpu().numpy().view(np.uint32), o.time.ravel().view(np.uint32))
    assert np.array_equal(d["rx"].cpu().numpy().view(np.uint16), o.refs_x.ravel())
    assert np.array_equal(d["ry"].cpu().numpy().view(np.uint16), o.refs_y.ravel())
    for k in SCHEDULE + WORK:
        assert st[k] == o.stats[k], k
    assert 0 < st["burned"] < 150 * 150
