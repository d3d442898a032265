"""Cells of more than 65,536 particles: a cutoff longer than the box makes the whole
system one cell. Their order is the stable sort's, as every cell's."""
import numpy as np
import pytest

import md_simulation_cuda_b200 as mdb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,Lx,Ly,cell_min", [(80000, 10.0, 10.0, 8.0), (150001, 20.0, 9.0, 9.0),
                                              (65537, 9.0, 9.0, 9.0)])
def test_order_is_stable(built, n, Lx, Ly, cell_min):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 1.0, (n, 2)) * [Lx, Ly]
    cell, perm, ncx, ncy = mdb.cell_build(pos, Lx, Ly, cell_min)
    c, p, nx, ny = po.cell_build(pos, Lx, Ly, cell_min)
    assert (ncx, ncy) == (nx, ny)
    assert np.array_equal(cell, c)
    assert np.array_equal(perm, p)
