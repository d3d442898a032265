"""The resident steps kernels (csrc/mdb_steps.cuh, mdb_band_steps.cuh) against one
kernel per phase.

Sizes at the edges of its blocks (64 slots with four lanes a slot up to 16,384
particles, 256 with one lane after that) and of what fits on the device, every
integrator and FIRE, and the list forms: shared columns, lists too long for
them, capacities that overflow into stencil scans, no lists at all. Every
result is bit for bit that of the per-phase kernels.
"""
import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _frame(n, aspect=1.0, rho=0.8, T=0.9, seed=5):
    f, Lx, Ly = wl.lattice_frame(n, rho, aspect, 0.6, T, seed=seed + n, jitter=0.1)
    return f, wl.config_dict(n, Lx, Ly, dt=0.002, T=0.9, barostat_mass=50.0, k_piston=100.0,
                             n_cap=n)


def _bits(sim):
    sim.sample_collect()
    f = sim.get_host_particles()
    o = sim.observables()
    return (f.tobytes(), o.t, o.Lx, o.Ly, o.xi, o.nph_area_momentum, o.nph_piston_velocity,
            o.nph_piston_force, o.last_instant_pressure, o.steps, o.rebuilds)


def _run(f, cfg, kernel, steps, **opt):
    sim = mdb.MDSimulation(cfg, frame=f, step_kernel=kernel, **opt)
    out = []
    sim.step_single_nose_hoover(nsteps=steps)
    out.append(_bits(sim))
    sim.step_single_NPH(1.2, nsteps=steps)
    out.append(_bits(sim))
    sim.step_single_NVE(nsteps=1)
    sim.step_single_NVE(nsteps=steps)
    out.append((_bits(sim), sim.cal_total_U()))  # reads the lists the run left
    sim.step_single_NPH_piston(0.8, nsteps=steps)
    out.append((_bits(sim), sim.cal_total_U()))
    sim.step_single_NVE(nsteps=5)  # back to the periodic box
    out.append(_bits(sim))
    return sim, out


@pytest.mark.parametrize("n,aspect", [(5, 1.0), (63, 1.0), (64, 1.0), (65, 2.0), (257, 1.0),
                                      (1023, 3.0), (16384, 1.0), (16385, 1.0), (75776, 2.0)])
def test_equals_per_phase(built, n, aspect):
    f, cfg = _frame(n, aspect)
    steps = 60 if n < 20000 else 30
    _, a = _run(f, cfg, mdb.STEPS_PER_PHASE, steps)
    sim, b = _run(f, cfg, mdb.STEPS_AUTO, steps)
    assert sim.schedule()["multi_step"] == 1
    assert a == b


def test_beyond_the_device(built):
    f, cfg = _frame(75777 + 256, 2.0)
    assert mdb.MDSimulation(cfg, frame=f).schedule()["multi_step"] == 0


@pytest.mark.parametrize("n,aspect,opt", [
    (75777 + 256, 2.0, {}), (80001, 0.01, {}), (100003, 60.0, {}), (151808, 1.0, {}),
    (230001, 3.0, {}), (90001, 1.0, dict(max_neighbors=15)), (90001, 1.0, dict(max_neighbors=-1)),
    (90001, 1.0, dict(skin=1.4))])
def test_staged_steps_equal_per_phase(built, n, aspect, opt):
    """Systems of several hundred blocks: the steps kernel over staged bands."""
    f, cfg = _frame(n, aspect)
    _, a = _run(f, cfg, mdb.STEPS_PER_PHASE, 30, **opt)
    _, b = _run(f, cfg, mdb.STEPS_AUTO, 30, **opt)
    assert a == b


@pytest.mark.parametrize("opt", [dict(max_neighbors=-1), dict(max_neighbors=14),
                                 dict(max_neighbors=400), dict(skin=0.12), dict(skin=1.4),
                                 dict(lanes=mdb.LANES_ONE),
                                 dict(lanes=mdb.LANES_ONE, max_neighbors=18)])
def test_list_forms(built, opt):
    f, cfg = _frame(1500, 1.5)
    _, a = _run(f, cfg, mdb.STEPS_PER_PHASE, 60, **opt)
    _, b = _run(f, cfg, mdb.STEPS_AUTO, 60, **opt)
    assert a == b


@pytest.mark.parametrize("n,precision,random", [(40, 0, False), (256, 2, True), (700, 0, True),
                                                (2048, 1, False), (30001, 0, False),
                                                (90001, 0, False), (160001, 2, False)])
def test_fire_equals_per_phase(built, n, precision, random):
    if random:
        f, L = wl.random_frame(n, 0.8, 0.5, seed=n)
        cfg = wl.config_dict(n, L, L, dt=0.001, T=0.0, n_cap=n)
    else:
        f, cfg = _frame(n, T=0.0)
    out = []
    for graphs in (False, True):  # False: one launch per phase
        r = mdb.EnergyMinimizer(cfg, use_graphs=graphs, fire_precision=precision).minimize_frame(
            f, 1e-5, 400, wl.fire_params())
        out.append((r.frame.tobytes(), r.steps, r.converged, r.max_force, r.energy_trace,
                    r.nonfinite))
    assert out[0] == out[1]
    assert np.isfinite(out[0][3])


@pytest.mark.parametrize("n,aspect", [(80001, 0.3), (151808, 2.0)])
def test_lists_change_no_bit(built, n, aspect):
    """Lists against stencil scans, through every integrator (forces of the same
    pairs in the same order)."""
    f, cfg = _frame(n, aspect)
    _, a = _run(f, cfg, mdb.STEPS_AUTO, 45)
    _, b = _run(f, cfg, mdb.STEPS_AUTO, 45, max_neighbors=-1)
    assert a == b
