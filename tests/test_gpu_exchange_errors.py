"""Exchanges of the resident steps kernels that give up.

MDB_EXCHANGE_POLLS=1@1 lets block 1 look once whether the others have arrived:
sooner or later it gives up an exchange that the others see through. That was the
launch's last exchange for a one-step call, whose other blocks then finish as
usual. The call has to end with an error all the same, and the error is final for
the handle.
"""
import pytest

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 30000])
def test_one_block_gives_up_the_last_exchange(built, monkeypatch, n):
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.5, 0.8, seed=n, jitter=0.1)
    cfg = wl.config_dict(n, Lx, Ly, dt=0.002, T=0.8)
    monkeypatch.setenv("MDB_EXCHANGE_POLLS", "1@1")
    sim = mdb.MDSimulation(cfg, frame=f)
    for k in range(200):  # (most likely the first call)
        try:
            sim.step_single_NVE()
            sim.synchronize()
        except mdb.MDBError:
            break
    else:
        pytest.fail("no call reported the exchange that gave up")
    for _ in range(3):
        with pytest.raises(mdb.MDBError):
            sim.step_single_NVE(nsteps=5)
            sim.synchronize()
    with pytest.raises(mdb.MDBError):
        sim.observables()
