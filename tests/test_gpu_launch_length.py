"""A launch of the steps kernels ends after about a millisecond of steps, so that
streams of higher priority get in."""
import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,low,high", [(1000000, 60, 5, 12), (300000, 60, 2, 4),
                                              (60000, 200, 3, 4), (4096, 200, 1, 2)])
def test_launches_of_one_call(built, n, steps, low, high):
    """low to high launches for a call of `steps` steps (95, 34, 15 and 6 us each)."""
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
    sim = mdb.MDSimulation(wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8), frame=f)
    sim.step_single_NVE()
    sim.synchronize()
    before = mdb.kernel_launches()
    sim.step_single_NVE(nsteps=steps)
    sim.synchronize()
    assert low <= mdb.kernel_launches() - before <= high


def test_served_systems_share_the_device(built):
    """A large system in a server's batch runs one kernel per phase."""
    n, steps = 100000, 64
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8)
    before = mdb.kernel_launches()
    with mdb.Server(device=0) as srv:
        rid = srv.submit_md(cfg, f, steps)
        srv.wait(rid)
        r = srv.result(rid)
    assert mdb.kernel_launches() - before >= 2 * steps
    sim = mdb.MDSimulation(cfg, frame=f)
    sim.step_single_nose_hoover(nsteps=steps)
    sim.sample_collect()
    assert np.array_equal(sim.get_host_particles()["pos"], r.frame["pos"])
