"""The two-pass line transforms of the grid kernel at every grid size they split (2-3-5 sizes up to 64), cubic and with
three different extents, against cuFFT in one field pass (direct + reciprocal field of given charges and dipoles)."""

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SIZES = [6, 8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64]
GRIDS = [(k, k, k) for k in SIZES] + [(6, 64, 9), (25, 60, 54), (64, 15, 20), (10, 27, 6)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_grid_kernel_matches_cufft(grid, precision):
    S = PKG.systems.waters(20, 9.0, seed=11, grid=grid, cutoff=4.4, tol=1e-6)
    rng = np.random.default_rng(5)
    d = rng.normal(0.0, 0.02, (S.n, 3))
    E = []
    for mode in (0, 3):
        eng = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=grid, order=6, predictor=0,
                                      precision=precision))
        eng.set_system(S)
        eng.set_transforms(mode)
        assert eng.transforms() == mode
        E.append(eng.field(S.pos, S.box, S.q, d))
        eng.close()
    # both transforms err by a few eps log2(points) of the spectrum (2^-53 or 2^-24, at most 18 levels), and the field
    # is the spectrum's derivative: 64 eps x 18 bounds the relative RMS difference
    eps = 2.0 ** -53 if precision == 0 else 2.0 ** -24
    assert np.linalg.norm(E[1] - E[0]) <= 64 * 18 * eps * np.linalg.norm(E[0])
