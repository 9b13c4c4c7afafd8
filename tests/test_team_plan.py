"""The rules that split a batch over the device (csrc/team_plan.hpp), on the
host: what the autotuner times for every number of jobs, and that the splits
use the CTAs they are given."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "team_plan.hpp"
using namespace propag;
extern "C" int plan_team(int n, const double *side, int ctas) { return team_size(std::vector<double>(side, side + n), ctas); }
extern "C" void plan_split(uint32_t n, int ctas, int team, uint32_t *out) {
  const GroupSplit g = group_split(n, ctas, team);
  out[0] = g.slots;
  out[1] = g.group;
}
extern "C" int plan_modes(uint32_t n, int ctas, int auto_team, int *out) {
  const std::vector<int> m = autotune_groups(n, ctas, auto_team);
  std::copy(m.begin(), m.end(), out);
  return (int)m.size();
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "p.cpp").write_text(SOURCE)
    so = d / "p.so"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(cuda, "include"),
                    "-I" + os.path.join(ROOT, "propag-hidalgo_b200", "csrc"), str(d / "p.cpp"), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))


def _split(plan, n, ctas, team):
    out = (C.c_uint32 * 2)()
    plan.plan_split(n, ctas, team, out)
    return tuple(out)


@pytest.mark.parametrize("ctas", [148, 132, 16])
@pytest.mark.parametrize("side", [128.0, 1024.0])
def test_autotuner_modes(plan, ctas, side):
    for n in list(range(1, 160)) + [256, 1000, 5000]:
        auto = plan.plan_team(n, (C.c_double * n)(*[side] * n), ctas)
        assert 2 <= auto <= ctas
        for auto_team in {auto, 0}:  # 0: the automatic mode is not one team a job's split
            out = (C.c_int * 16)()
            count = plan.plan_modes(n, ctas, auto_team, out)
            modes = list(out)[:count]
            assert modes[0] == 0 and all(m <= -2 for m in modes[1:])
            splits = [_split(plan, n, ctas, -m) for m in modes[1:]] + (
                [_split(plan, n, ctas, auto_team)] if auto_team else [])
            assert len(set(splits)) == len(splits), n  # nothing is timed twice
            if ctas // n >= 2:  # a team per job is among them
                assert (n, ctas // n) in splits, n
            for team in (24, 16, 8, 4):
                if team <= ctas:
                    assert _split(plan, n, ctas, team) in splits, (n, team)
            for slots, group in splits:
                assert 1 <= slots <= n and group >= 2 and slots * group <= ctas


def _alike(sides, teams, ctas):
    """The end of a batch whose jobs take their mean time, on teams of equal size."""
    ends = [0.0] * teams
    for s in sorted(sides, reverse=True):
        i = ends.index(min(ends))
        ends[i] += 7.6 * s + 0.229 * s * s / (ctas // teams)
    return max(ends)


@pytest.mark.parametrize("side", [64.0, 150.0, 400.0, 700.0, 1024.0, 2000.0])
def test_team_size_where_jobs_are_alike(plan, side):
    """The teams chosen for differing jobs lose at most a factor 1.85 where the jobs
    are alike, of any number (1.9 and more for 5 to 40 jobs before)."""
    ctas = 148
    for n in list(range(1, 80)) + [100, 148, 200]:
        team = plan.plan_team(n, (C.c_double * n)(*[side] * n), ctas)
        slots, group = _split(plan, n, ctas, team)
        best = min(_alike([side] * n, t, ctas) for t in range(1, min(n, ctas // 2) + 1))
        assert _alike([side] * n, slots, ctas) <= 1.85 * best, (n, slots)


def test_team_size_of_uneven_batches(plan):
    """A few large jobs among many small ones: few teams, so that the large ones
    get many CTAs."""
    ctas = 148
    for sides in ([4096.0] + [128.0] * 100, [3000.0] * 2 + [500.0] * 10, [2048.0] * 3 + [256.0] * 40):
        team = plan.plan_team(len(sides), (C.c_double * len(sides))(*sides), ctas)
        assert team >= 37
    assert plan.plan_team(1, (C.c_double * 1)(4096.0), ctas) == ctas
