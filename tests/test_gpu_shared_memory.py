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


def box(grid, precision, molecules=40, seed=5, **kw):
    S = PKG.systems.waters(molecules, (molecules / 0.0334) ** (1 / 3), seed=seed, grid=grid, cutoff=4.0, tol=1e-8)
    e = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=S.grid, order=6, tol=1e-8, max_iter=500, peek=0.0,
                                predictor=0, ke=PKG.systems.KE_DEFAULT, precision=precision, **kw))
    e.set_system(S)
    return S, e


@pytest.mark.parametrize("precision,mode,pme", [(0, None, 0), (0, 3, 0), (1, None, 0), (1, 1, 0), (1, 3, 0),
                                                (1, 4, 0), (1, 0, 1), (1, 4, 1)])
def test_two_engines_of_different_grids(precision, mode, pme):
    """An engine computes what it computes alone while a second one, of a smaller grid on the same kernel instances, was set
    up after it and while it lives (the shared-memory limit belongs to the kernel, not to the engine)."""
    out = []
    for beside in (False, True):
        S, a = box((48, 54, 60), precision)
        if beside:
            T, b = box((24, 30, 36), precision, molecules=24, seed=6)
        for e in (a, b) if beside else (a,):
            if mode is not None:
                e.set_transforms(mode)
                assert e.transforms() == mode
            e.set_pme_kernels(pme)
        r = a.compute(S.pos, S.box)
        if beside:
            b.compute(T.pos, T.box)
            r = a.compute(S.pos, S.box)
            b.close()
        out.append(r)
        a.close()
    # (the same kernels on the same inputs; float and double atomics aside, the same bits)
    lim = 1e-12 if precision == 0 else 1e-6
    assert abs(out[0].energy - out[1].energy) <= lim * abs(out[0].energy)
    assert np.linalg.norm(out[0].forces - out[1].forces) <= lim * np.linalg.norm(out[0].forces)
