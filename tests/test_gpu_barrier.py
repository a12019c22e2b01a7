"""The failure path of the grid transforms' barriers, exercised without a GPU fault: a block waits at a barrier
that expects one block more than the launch has, so nothing ever ends its wait.  The wait gives up after its
bounded number of polls (about a second), sets the error flag the host reads, and returns; the context stays
usable and the next evaluation is correct."""

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu


def test_grid_barrier_wait_gives_up_and_reports():
    S = PKG.systems.water216()
    eng = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=S.grid, order=S.order, tol=1e-8,
                                  precision=PKG.FP64))
    eng.set_system(S)
    before = eng.compute(S.pos, S.box).energy
    gave_up, seconds = eng.probe_barrier_timeout()
    assert gave_up
    assert 1e-3 < seconds < 10.0
    after = eng.compute(S.pos, S.box).energy
    assert np.isfinite(after) and abs(after - before) <= 1e-12 * abs(before)


@pytest.mark.parametrize("precision,mode,grid", [(0, 3, (20, 20, 20)), (1, 3, (20, 20, 20)), (1, 4, (20, 20, 20)),
                                                 (0, 3, (18, 20, 24))])
def test_launches_after_a_barrier_gave_up_do_not_wait(precision, mode, grid):
    """Grid-kernel launches that find the error flag set return at once, in place of a second at each of their barriers; the
    next evaluation is unchanged (the sources that the self-test's spread left on the fixed-point grid are gone)."""
    S = PKG.systems.water216()
    eng = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=grid, order=S.order, tol=1e-8, predictor=0,
                                  precision=precision))
    eng.set_system(S)
    eng.set_transforms(mode)
    assert eng.transforms() == mode
    before = eng.compute(S.pos, S.box)
    gave_up, _ = eng.probe_barrier_timeout()   # (False when a later launch came to its barrier)
    assert gave_up
    after = eng.compute(S.pos, S.box)
    lim = 1e-12 if precision == 0 else 1e-6
    assert abs(after.energy - before.energy) <= lim * abs(before.energy)
    assert np.linalg.norm(after.forces - before.forces) <= lim * np.linalg.norm(before.forces)
    eng.close()
