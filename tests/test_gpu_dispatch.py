"""The transforms that an engine takes until the caller chooses, and the persistent kernel at the edges of its slot split (fewer
atoms than blocks, one slot a block, a remainder) and from each initial guess."""

import threading

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu


def engine(S, precision=1, tol=1e-8, zero_guess=False, order=6, predictor=0, **kw):
    e = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=S.grid, order=order, tol=tol, max_iter=500, peek=0.0,
                                predictor=predictor, ke=PKG.systems.KE_DEFAULT, precision=precision,
                                zero_guess=zero_guess, **kw))
    e.set_system(S)
    return e


def water(molecules, K=None):
    L = (molecules / 0.0334) ** (1 / 3)
    K = K or max(8, PKG.systems.fft_size(L))
    return PKG.systems.waters(molecules, L, seed=molecules, grid=(K, K, K), cutoff=min(9.0, L / 2), tol=1e-8)


@pytest.mark.parametrize("molecules", [8, 49, 50, 99, 198, 443])   # 24, 147, 150, 297, 594, 1329 atoms on 148 blocks
@pytest.mark.parametrize("zero_guess", [False, True])
def test_persistent_kernel_slot_split(molecules, zero_guess):
    """Against the graph loop with the grid kernel: the same iterations, and results that differ by the rounding of float
    sums in another order (a few 2^-24 over sums whose terms cancel to a tenth: 3e-6)."""
    S = water(molecules)
    out = []
    for mode in (3, 4):
        e = engine(S, zero_guess=zero_guess)
        e.set_transforms(mode)
        assert e.transforms() == mode
        r = e.compute(S.pos, S.box)
        out.append((r.energy, r.forces, e.induced_dipoles(), r.iterations, r.strain))
        x, _ = e.solve(out[-1][2], tol=1e-8)   # the adjoint's operator, from the zero guess
        out[-1] += (x,)
        e.close()
    a, b = out
    assert abs(a[3] - b[3]) <= 1
    assert abs(a[0] - b[0]) <= 3e-6 * abs(a[0])
    for k in (1, 2, 4, 5):
        assert np.linalg.norm(a[k] - b[k]) <= 3e-6 * np.linalg.norm(a[k]), k


def test_persistent_kernel_beyond_shared_memory():
    """105000 atoms, whose state the blocks' shared memory does not hold: the rule takes the grid kernel, and a choice of the
    persistent kernel still runs it, with the results of the graph loop (as above; the zero guess and the solve's)."""
    S = water(35000, K=64)
    S.tol = 1e-6
    out = []
    for mode in (3, 4):
        e = engine(S, tol=1e-6)
        assert e.transforms() == 3
        e.set_transforms(mode)
        assert e.transforms() == mode
        r = e.compute(S.pos, S.box)
        x, _ = e.solve(e.induced_dipoles(), tol=1e-6)
        out.append((r.energy, r.iterations, r.forces, r.strain, x))
        e.close()
    a, b = out
    assert abs(a[1] - b[1]) <= 1
    assert abs(a[0] - b[0]) <= 3e-6 * abs(a[0])
    for k in (2, 3, 4):
        assert np.linalg.norm(a[k] - b[k]) <= 3e-6 * np.linalg.norm(a[k]), k


def test_persistent_kernel_predicted_steps():
    """Steps of a moving system, each guess of the predictor in turn (none, the last solution, mu3, mu4), with a kept list."""
    S = water(120)
    rng = np.random.default_rng(2)
    phase = rng.uniform(0, 2 * np.pi, S.pos.shape)
    traj = [S.pos + 0.005 * np.sin(2 * np.pi * t / 60 + phase) for t in range(7)]
    runs = []
    for mode in (3, 4):
        e = engine(S, predictor=2, skin=0.1)
        e.set_transforms(mode)
        runs.append([e.compute(p, S.box) for p in traj])
        e.close()
    for a, b in zip(*runs):
        assert abs(a.iterations - b.iterations) <= 1
        assert abs(a.energy - b.energy) <= 3e-6 * abs(a.energy)
        assert np.linalg.norm(a.forces - b.forces) <= 3e-6 * np.linalg.norm(a.forces)


def test_transforms_without_a_choice():
    S = water(64, K=16)
    assert engine(S).transforms() == 4                       # mixed, one system, order 6
    assert engine(S, precision=0).transforms() == 3          # FP64: the grid kernel
    assert engine(S, order=5).transforms() == 3
    assert engine(S, polarizable=False).transforms() == 3
    assert engine(water(64, K=14)).transforms() == 0         # 14 = 2 x 7
    e = engine(S)
    e.set_pme_kernels(2)                                     # the caller's spread and gather run in the loop
    assert e.transforms() == 3 and e.pme_kernels() == 2
    e.set_transforms(0)                                      # the caller's choice stands
    assert e.transforms() == 0
    b = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=S.grid, order=6, precision=1))
    b.set_systems([S, S])
    assert b.transforms() == 0                               # batches


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("grid", [(6, 6, 6), (10, 12, 15), (24, 30, 36), (16, 16, 20)])
def test_grids_without_an_instance_keep_cufft(grid, precision):
    """The general instances of the persistent and the grid kernel are slower than cuFFT: only a choice takes them."""
    S = PKG.systems.waters(20, 9.0, seed=3, grid=grid, cutoff=4.4, tol=1e-6)
    e = engine(S, precision=precision)
    assert e.transforms() == 0
    for mode in (3, 4):
        e.set_transforms(mode)
        assert e.transforms() == (mode if mode == 3 or precision == 1 else 0)
    e.close()


def test_pair_lanes_of_the_rule():
    """FP64 with few lanes in the pair passes keeps cuFFT until the caller chooses; mixed does not depend on them."""
    S = water(64, K=16)
    for precision, modes in ((0, (0, 0, 3, 3)), (1, (4, 4, 4, 4))):
        e = engine(S, precision=precision)
        for lanes, mode in zip((4, 8, 16, 32), modes):
            e.set_pair_lanes(lanes)
            assert e.transforms() == mode
        e.set_transforms(3)
        e.set_pair_lanes(8)
        assert e.transforms() == 3   # (a choice stands)
        e.close()


@pytest.mark.parametrize("atoms,K,precision,mode", [(85500, 64, 1, 4), (87000, 64, 1, 3), (93000, 48, 1, 4), (98304, 48, 1, 3),
                                                    (12000, 64, 0, 3), (12300, 64, 0, 0), (39000, 60, 0, 3)])
def test_atom_counts_of_the_rule(atoms, K, precision, mode):
    e = PKG.Engine(PKG.Settings(cutoff=0.9, beta=3.5, grid=(K, K, K), order=6, precision=precision))
    e.set_atoms(np.zeros(atoms), np.full(atoms, 0.07), np.full(atoms, 1e-3))
    assert e.transforms() == mode
    e.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_other_covalent_dipoles_after_an_evaluation(precision):
    """A second set_covalent with fewer and then with more dipoles than the evaluation's graph was captured with gives what a
    fresh engine gives (the same kernels on the same inputs: FP64 atomics aside, the same bits)."""
    S = water(30)
    half = len(S.cov_atom) // 2
    e = PKG.Engine(PKG.Settings(cutoff=S.cutoff, beta=S.beta, grid=S.grid, order=6, tol=1e-8, max_iter=500, peek=0.0,
                                predictor=0, ke=PKG.systems.KE_DEFAULT, precision=precision, skin=0.0))
    e.set_atoms(S.q, S.radius, S.alpha)
    for m in (half, 2, len(S.cov_atom)):
        e.set_covalent(S.cov_atom[:m], S.cov_partner[:m], S.cov_strength[:m])
        for _ in range(2):
            r = e.compute(S.pos, S.box)
        fresh = engine(S, precision=precision, skin=0.0)
        fresh.set_covalent(S.cov_atom[:m], S.cov_partner[:m], S.cov_strength[:m])
        f = fresh.compute(S.pos, S.box)
        assert abs(r.energy - f.energy) <= 1e-12 * abs(f.energy)
        assert np.linalg.norm(r.forces - f.forces) <= 1e-12 * np.linalg.norm(f.forces)


GRIDS = [(6, 6, 6), (24, 30, 36), (25, 60, 54), (64, 15, 20), (10, 27, 6), (8, 64, 64), (15, 9, 25)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_general_instances_against_cufft(grid, precision):
    """Whole evaluations by the instances for any grid (three different extents, odd ones, few planes of many lines and many
    of few): the grid kernel with its energy variant and the persistent kernel against cuFFT's chain, and the solve of another
    right-hand side.  Mixed: the rounding of float sums in another order, as above; FP64: 64 eps x 18 levels (1.3e-13) of the
    transforms, carried through some ten iterations and the strain's cancelling terms (100 times that)."""
    S = PKG.systems.waters(20, 9.0, seed=11, grid=grid, cutoff=4.4, tol=1e-8)
    lim = 1.3e-11 if precision == 0 else 3e-6
    out = []
    for mode in (0, 3, 4) if precision == 1 else (0, 3):
        e = engine(S, precision=precision)
        e.set_transforms(mode)
        assert e.transforms() == mode
        r = e.compute(S.pos, S.box)
        mu = e.induced_dipoles()
        x, _ = e.solve(np.roll(mu, 1, axis=0), tol=1e-8)
        out.append((r.energy, r.iterations, r.forces, r.strain, mu, x))
        e.close()
    for b in out[1:]:
        a = out[0]
        assert abs(a[1] - b[1]) <= 1
        assert abs(a[0] - b[0]) <= lim * abs(a[0])
        for k in (2, 3, 4, 5):
            assert np.linalg.norm(a[k] - b[k]) <= lim * np.linalg.norm(a[k]), k


def test_engines_in_two_threads():
    """Engines in threads of their own, each with its cooperative kernels (the persistent one in a compiled and the general
    instance, the FP64 grid kernel): every evaluation is what the engine computes alone."""
    cases = [(water(300), 1, None), (water(120), 0, None),
             (PKG.systems.waters(40, 10.7, seed=4, grid=(24, 30, 36), cutoff=5.0, tol=1e-8), 1, 4)]
    engines, alone = [], []
    for S, precision, mode in cases:
        e = engine(S, precision=precision)
        if mode is not None:
            e.set_transforms(mode)
        engines.append(e)
        alone.append(e.compute(S.pos, S.box))
    assert [e.transforms() for e in engines] == [4, 3, 4]
    wrong = []

    def work(k):
        S, precision, _ = cases[k]
        lim = 1e-11 if precision == 0 else 1e-6
        try:
            for _ in range(60):
                r = engines[k].compute(S.pos, S.box)
                if not (abs(r.energy - alone[k].energy) <= lim * abs(alone[k].energy) and
                        np.linalg.norm(r.forces - alone[k].forces) <= lim * np.linalg.norm(alone[k].forces)):
                    wrong.append((k, r.energy, alone[k].energy))
        except Exception as ex:   # (a thread's error is the test's)
            wrong.append((k, repr(ex)))

    for pair in ((0, 1), (0, 2), (0, 1, 2)):
        threads = [threading.Thread(target=work, args=(k,)) for k in pair]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong, (pair, wrong[:3])
    for e in engines:
        e.close()


def test_kernel_launches_counted():
    """The launch count of each solve: without a skin 9 to the records, the permanent field 3, the persistent kernel 1 and the
    final pass 4; the graph loop 3 + 4 + 2, 5 an iteration and 6; with cuFFT the fixed-point grid's conversion in each pass.
    With the refinement the loop's kernels run whatever the mode."""
    S = water(64, K=16)
    for mode, refine, count in ((4, False, lambda it: 17), (3, False, lambda it: 24 + 5 * it), (0, False, lambda it: 27 + 6 * it),
                                (4, True, lambda it: 24 + 5 * it), (3, True, lambda it: 24 + 5 * it)):
        e = engine(S, tol=1e-6, skin=0.0, refine=refine)
        e.set_transforms(mode)
        r = e.compute(S.pos, S.box)
        assert e.kernel_launches() == count(r.iterations), (mode, refine)
        e.close()
