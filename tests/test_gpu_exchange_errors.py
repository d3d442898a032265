"""Exchanges of the resident steps kernels that give up, and ones that must not.

MDB_EXCHANGE_POLLS=4096@1 lets block 1 wait for one arrival more than there are: it
gives the last exchange of a launch up, a millisecond or so after the other blocks
have seen it through and finished as usual. The call has to end with an error all the
same, and the error is final for the handle. Blocks that are only slow are waited
for.
"""
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 30000, 75000])
def test_one_block_gives_up_the_last_exchange(built, monkeypatch, n):
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8)
    monkeypatch.setenv("MDB_EXCHANGE_POLLS", "4096@1")
    sim = mdb.MDSimulation(cfg, frame=f)
    with pytest.raises(mdb.MDBError):
        sim.step_single_NVE()
        sim.synchronize()
    for _ in range(3):
        with pytest.raises(mdb.MDBError):
            sim.step_single_NVE(nsteps=5)
            sim.synchronize()
    with pytest.raises(mdb.MDBError):
        sim.observables()


def test_slow_blocks_are_waited_for(built, monkeypatch):
    """A strip that its barostat squeezes below three cells turns into an all-pairs
    system in the middle of a run, with force phases of some 60 ms: 625 chunks on 313
    blocks, two each but for one, which waits half of that, against some 3 ms that two
    waits of 8,192 polls take. (A piece of a scan is marked every 0.2 ms.)"""
    n, Ly = 159900, 8.87
    f, Lx, Ly = wl.lattice_frame(n, 0.8, n / 0.8 / Ly ** 2, 0.5, 0.8, seed=n, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8, barostat_mass=2.5e-5, n_cap=n)
    out = []
    for kernel in (mdb.STEPS_PER_PHASE, mdb.STEPS_AUTO):
        monkeypatch.setenv("MDB_EXCHANGE_POLLS", "8192")
        sim = mdb.MDSimulation(cfg, frame=f, step_kernel=kernel)
        sim.step_single_NPH(50.0, nsteps=30)
        sim.sample_collect()
        o = sim.observables()
        assert o.Ly < 8.85 and o.rebuilds > 1
        out.append((sim.get_host_particles().tobytes(), o.Lx, o.Ly, o.steps, o.rebuilds))
    assert out[0] == out[1]
