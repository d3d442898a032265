"""Neighbour lists of staged bands (csrc/mdb_band.cuh) where whole rows of cells
do not fit one, and of the systems that bands do not fit at all.

A box three or four cells high has rows longer than a staged band, and a
lattice's rows of cells are so unequal that three of them and their neighbours
are. Their chunks take stretches of rows: every slot keeps its list (the batch
counts the ones that lost it), and the results are those of the per-phase kernels
and of stencil scans, bit for bit.
"""
import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _strip(n, Ly, rho=0.8, **cfg):
    """A lattice in a box of height Ly (cells are 2.95 high, for FIRE 2.7)."""
    f, Lx, Ly = wl.lattice_frame(n, rho, n / rho / Ly ** 2, 0.5, 0.8, seed=n, jitter=0.1)
    return f, wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8, barostat_mass=50.0, k_piston=100.0,
                             n_cap=n, **cfg)


@pytest.mark.parametrize("n,Ly", [(9000, 9.2), (9001, 12.5), (20011, 14.7)])
@pytest.mark.parametrize("fire", [False, True])
def test_low_boxes_keep_their_lists(built, n, Ly, fire):
    f, cfg = _strip(n, Ly)
    b = mdb.Batch()
    for _ in range(2):
        if fire:
            b.add_fire(cfg, f, 1e-9, 1000, wl.fire_params())
        else:
            b.add_md(cfg, f, mdb.JOB_NVT, 40)
    b.run(0 if fire else -1)
    for k in range(2):
        assert b.system_stats(k)[1] == 0  # (rebuilds, slots without a list)


@pytest.mark.parametrize("n,aspect", [(16384, 1.0), (16385, 1.0), (40000, 1.0), (25600, 0.4)])
def test_lattices_keep_their_lists(built, n, aspect):
    f, Lx, Ly = wl.lattice_frame(n, 0.8, aspect, 0.5, 0.8, seed=n, jitter=0.1)
    b = mdb.Batch()
    for _ in range(2):
        b.add_md(wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8), f, mdb.JOB_NVT, 40)
    b.run(0)
    for k in range(2):
        assert b.system_stats(k) == (1, 0)  # one rebuild, no slot without a list


def _run(f, cfg, steps, **opt):
    sim = mdb.MDSimulation(cfg, frame=f, **opt)
    out = []
    for step in (lambda: sim.step_single_nose_hoover(nsteps=steps),
                 lambda: sim.step_single_NPH(1.2, nsteps=steps),
                 lambda: sim.step_single_NPH_piston(0.8, nsteps=steps),
                 lambda: sim.step_single_NVE(nsteps=5)):
        step()
        sim.sample_collect()
        o = sim.observables()
        out.append((sim.get_host_particles().tobytes(), o.Lx, o.Ly, o.xi, o.rebuilds,
                    sim.cal_total_U()))
    return out


@pytest.mark.parametrize("n,Ly", [(80001, 9.2), (80003, 12.5), (100003, 16.0)])
def test_low_boxes_in_the_steps_kernel(built, n, Ly):
    f, cfg = _strip(n, Ly)
    a = _run(f, cfg, 30)
    assert a == _run(f, cfg, 30, step_kernel=mdb.STEPS_PER_PHASE)
    assert a == _run(f, cfg, 30, max_neighbors=-1)


@pytest.mark.parametrize("cutoff,nbr", [(7.0, 190), (9.0, 320), (3.0, None)])
def test_long_cutoffs_keep_their_lists(built, cutoff, nbr):
    """Cells too full for a band: lists of slot offsets instead of stencil scans."""
    n = 9000
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=3, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8, cutoff=cutoff)
    b = mdb.Batch(max_neighbors=nbr)
    for _ in range(2):
        b.add_md(cfg, f, mdb.JOB_NVT, 40)
    b.run(0)
    assert b.system_stats(1)[0] == 1  # one rebuild, whichever lists it ended with
    b.run()
    assert b.system_stats(1)[1] == 0
    sim = mdb.MDSimulation(cfg, frame=f, max_neighbors=nbr, lanes=mdb.LANES_ONE)
    sim.step_single_nose_hoover(nsteps=40)
    sim.sample_collect()
    for k in range(2):
        assert np.array_equal(sim.get_host_particles()["pos"], b.frame(k)["pos"])


@pytest.mark.parametrize("n,Ly,cutoff", [(80001, 8.0, 2.5), (90001, 300.0, 8.0)])
def test_large_systems_without_bands(built, n, Ly, cutoff):
    """All pairs, and a long cutoff: the forms agree bit for bit."""
    f, cfg = _strip(n, Ly, cutoff=cutoff)
    steps = 3 if Ly < 8.85 else 20
    a = _run(f, cfg, steps, max_neighbors=240)
    assert a == _run(f, cfg, steps, max_neighbors=240, step_kernel=mdb.STEPS_PER_PHASE)
    assert a == _run(f, cfg, steps, max_neighbors=-1)


def test_fire_with_a_long_cutoff(built):
    """FIRE on lists of slot offsets: a batch against quenches by themselves."""
    res = []
    for n in (3000, 3333):
        f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.2)
        res.append((f, wl.config_dict(n, Lx, Ly, dt=0.001, T=0.0, cutoff=7.0, n_cap=n)))
    b = mdb.Batch(max_neighbors=190)
    for f, cfg in res:
        b.add_fire(cfg, f, 1e-5, 200, wl.fire_params())
    b.run()
    for k, (f, cfg) in enumerate(res):
        a = mdb.EnergyMinimizer(cfg).minimize_frame(f, 1e-5, 200, wl.fire_params())
        r = b.fire_result(k)
        assert a.steps == r.steps and a.max_force == r.max_force
        assert np.array_equal(a.frame["pos"], r.frame["pos"])


def test_clustered_frames_keep_their_lists(built):
    """A droplet of a high density in a large empty box: the mean density says that its
    chunks fit, the frame's own count that they don't."""
    n = 9000
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.1, seed=4, jitter=0.02)
    f["pos"] += 3.0 * Lx
    cfg = wl.config_dict(n, 7.0 * Lx, 7.0 * Ly, dt=0.0005, T=0.1, cutoff=7.0)
    b = mdb.Batch(max_neighbors=190)
    for _ in range(2):
        b.add_md(cfg, f, mdb.JOB_NVE, 20)
    b.run(0)
    assert b.system_stats(0) == (1, 0)
    b.run()
    sim = mdb.MDSimulation(cfg, frame=f, max_neighbors=190, lanes=mdb.LANES_ONE)
    sim.step_single_NVE(nsteps=20)
    sim.sample_collect()
    assert np.array_equal(sim.get_host_particles()["pos"], b.frame(1)["pos"])
