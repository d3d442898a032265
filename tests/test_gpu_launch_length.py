"""A launch of the steps kernels ends after about a millisecond of steps, so that
streams of higher priority get in."""
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
