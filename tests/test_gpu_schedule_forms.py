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


@pytest.mark.parametrize("form", ["bands", "lists"])
def test_tuned_batches_are_bit_identical(built, tmp_path, monkeypatch, form):
    """MD batches with staged bands and with lists of slot offsets: the velocities and
    accelerations that the timed force phases change are put back."""
    monkeypatch.setenv("MDB_SCHEDULE_CACHE", str(tmp_path / "schedule.txt"))
    out = []
    for tune in (False, True):
        b = mdb.Batch(autotune=tune, max_neighbors=None if form == "bands" else 200)
        for n in (700, 3001, 9000):
            f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
            b.add_md(wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8,
                                    cutoff=2.5 if form == "bands" else 7.0),
                     f, mdb.JOB_NVT, 60)
        b.run()
        assert b.schedule()["tuned"] == int(tune)
        out.append([b.frame(k).tobytes() for k in range(3)])
    assert out[0] == out[1]
