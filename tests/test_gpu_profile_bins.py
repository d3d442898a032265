"""Profiles at the bin counts where their kernels differ: fewer bins than a
thread's window, bins finer than the window reaches, sizes off the warp and
block, a system scanned as a whole, a walled axis. Against the oracle: counts
equal, pressure bins within 1e-5 of the largest (FP32 pair terms)."""
import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb,walled", [(30, 5, False), (1000, 1, False), (1001, 2, False),
                                         (3000, 3, False), (3001, 7, False), (3000, 40, False),
                                         (3017, 300, False), (2000, 12, True), (2000, 90, True)])
def test_profiles_against_the_oracle(built, n, nb, walled):
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.5, 0.6, 0.8, seed=300 + n, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.001, T=0.8, barostat_mass=1e4, k_piston=100.0)
    sim = mdb.MDSimulation(cfg, frame=f)
    if walled:
        sim.step_single_NPH_piston(0.5, nsteps=5)
    else:
        sim.step_single_nose_hoover(nsteps=20)
    sim.sample_collect()
    g = sim.get_host_particles()
    a, b = po.n_profile(g["pos"], g["type"], sim.get_Lx(), nb)
    assert np.array_equal(sim.get_N_profile(nb), np.concatenate([a, b]))
    ref = np.concatenate(po.pressure_profile(cfg, g["pos"], g["vel"], g["type"], sim.get_Lx(),
                                             sim.get_Ly(), nb, periodic_y=0 if walled else 1))
    got = sim.get_pressure_profile(nb)
    assert np.max(np.abs(got - ref)) <= 1e-5 * np.max(np.abs(ref))
    assert np.array_equal(got, sim.get_pressure_profile(nb))
