"""The autotuner and the kernels that a handle runs (see test_gpu_schedule.py)."""
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _sim(n, **opt):
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
    return mdb.MDSimulation(wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8), frame=f, **opt)


def test_schedules_of_other_kernels_do_not_match(built, tmp_path, monkeypatch):
    """Sizes of one bucket on either side of what the resident steps kernel holds, and
    one kernel per phase."""
    monkeypatch.setenv("MDB_SCHEDULE_CACHE", str(tmp_path / "schedule.txt"))
    cached = [_sim(70000, autotune=True).schedule()["from_cache"],
              _sim(80000, autotune=True).schedule()["from_cache"],
              _sim(80000, autotune=True, step_kernel=mdb.STEPS_PER_PHASE).schedule()["from_cache"],
              _sim(70000, autotune=True).schedule()["from_cache"]]
    assert cached == [0, 0, 0, 1]


@pytest.mark.parametrize("n,extra", [(900, 0), (20000, 0), (100000, 16)])
def test_only_what_steps_read_is_timed(built, tmp_path, monkeypatch, n, extra):
    """Launches at creation beyond those of an untuned handle: none for the resident
    steps kernel, four candidates of the prefetch depth (one launch and three) over
    staged bands."""
    monkeypatch.setenv("MDB_SCHEDULE_CACHE", str(tmp_path / "schedule.txt"))
    count = []
    for tune in (False, True):
        before = mdb.kernel_launches()
        sim = _sim(n, autotune=tune)
        count.append(mdb.kernel_launches() - before)
        assert sim.schedule()["tuned"] == int(tune)
    assert count[1] - count[0] == extra
