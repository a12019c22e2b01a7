"""Engines whose kernels need different amounts of shared memory, alone and beside each other."""

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu


def settings(grid, cutoff=0.9, beta=3.5, **kw):
    return PKG.Settings(cutoff=cutoff, beta=beta, grid=grid, order=6, max_iter=500, peek=0.0, predictor=0,
                        ke=PKG.systems.KE_DEFAULT, precision=PKG.MIXED, **kw)


@pytest.mark.parametrize("atoms,K", [(103400, 64), (111200, 48), (116900, 32)])
def test_setup_where_the_static_part_decides(atoms, K):
    """The persistent kernel's state for this many atoms fits a block's shared memory without the kernel's static 1.5 KB and
    not with it: the engine is set up all the same, on the grid kernel."""
    e = PKG.Engine(settings((K, K, K)))
    e.set_atoms(np.zeros(atoms), np.full(atoms, 0.07), np.full(atoms, 1e-3))
    assert e.transforms() == 3
    e.close()
