"""Systems that lose their numbers end in bounded time, whichever way they do."""
import time

import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [1e300, np.inf, -np.inf, np.nan])
def test_piston_with_positions_beyond_all_numbers(built, value):
    """The walled y axis is not wrapped: in a box a few cells wide, y positions that
    are infinite (or are as the pair loop's FP32) put 130,000 particles into each
    cell of one row. Scanning them takes 290 ms a step, 10 steps 2.9 s; here 0.2 s
    are left, most of them the sort of finite ones."""
    n = 400000
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 0.0002, 0.5, 0.8, seed=1, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8, k_piston=100.0, n_cap=n)
    f["vel"][:, 1] = value
    sim = mdb.MDSimulation(cfg, frame=f)
    sim.sample_collect()
    t = time.perf_counter()
    sim.step_single_NPH_piston(1.0, nsteps=10)
    sim.sample_collect()
    assert time.perf_counter() - t < 1.0
    assert sim.observables().nonfinite == (0 if value == 1e300 else 1)
