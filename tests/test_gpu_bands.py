"""Staged bands (csrc/mdb_band.cuh): the force phase and list build of batches
and of systems beyond the resident steps kernel.

Box shapes that reach every form of a chunk's band (whole rows, three row
pieces, two pieces of four rows, both periodic edges, the walled axis), ragged
sizes, list overflow and no lists. A system in a batch is bit for bit the one
in a simulation handle (other kernels), and large systems agree with the
oracle's forces.
"""
import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

SHAPES = [(40, 1.0), (255, 1.0), (256, 2.0), (257, 0.5), (1000, 1.0), (3000, 6.0), (3000, 0.15),
          (5003, 1.0), (9000, 0.02), (9001, 60.0), (20000, 2.0)]


@pytest.mark.parametrize("max_nbr", [None, 15, -1])
def test_batch_equals_simulation(built, max_nbr):
    frames = []
    for k, (n, aspect) in enumerate(SHAPES):
        f, Lx, Ly = wl.lattice_frame(n, 0.8, aspect, 0.5, 0.8, seed=70 + k, jitter=0.1)
        frames.append((f, wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8)))
    b = mdb.Batch(max_neighbors=max_nbr)
    for f, cfg in frames:
        b.add_md(cfg, f, mdb.JOB_NVT, 60)
    b.run()
    for k, (f, cfg) in enumerate(frames):
        sim = mdb.MDSimulation(cfg, frame=f, lanes=mdb.LANES_ONE)
        sim.step_single_nose_hoover(nsteps=60)
        sim.sample_collect()
        g = sim.get_host_particles()
        h = b.frame(k)
        for name in ("pos", "vel", "acc", "type"):
            assert np.array_equal(g[name], h[name]), (SHAPES[k], name)


@pytest.mark.parametrize("n,aspect,periodic", [(80000, 1.0, True), (90001, 7.0, True),
                                               (90001, 0.01, True), (100003, 90.0, True),
                                               (80000, 2.0, False), (100003, 0.05, False)])
def test_large_systems_against_the_oracle(built, n, aspect, periodic):
    f, Lx, Ly = wl.lattice_frame(n, 0.8, aspect, 0.5, 0.8, seed=n, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8)
    acc, U, W = mdb.compute_forces(cfg, f, Lx, Ly, periodic_y=periodic)
    F, Uo, _ = po.forces(cfg, f["pos"], f["type"], Lx, Ly, periodic_y=int(periodic),
                         cells=True)
    assert np.linalg.norm(acc - F) <= 1e-5 * np.linalg.norm(F)
    assert abs(U - Uo) <= 1e-6 * abs(Uo)


@pytest.mark.parametrize("n", [100003, 400001])
def test_nonfinite_system_ends(built, n):
    """A system that has lost its numbers (all positions in one cell) still steps
    in bounded time and says so."""
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
    f["vel"] = np.nan
    sim = mdb.MDSimulation(wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8), frame=f)
    sim.step_single_NVE(nsteps=3)
    assert sim.observables().nonfinite == 1
