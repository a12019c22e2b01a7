"""Performance cases of the pGM engine: what its users have it do, over the range of sizes they do it at.

A case is a dict of plain values:

    call        the public entry point that a pass goes through (below)
    system      "water", "dimethylphenol" (liquids at their densities) or "triclinic" (waters in a triclinic box)
    molecules   molecules of the system (of the largest box, for a batch)
    systems     boxes of a batch (1: a single-system engine)
    precision   "mixed" or "fp64"
    tol         the dipole solver's tolerance
    skin        the Verlet list's skin [nm]: 0 builds the pair list in every evaluation
    lanes, transforms
                what Engine.set_pair_lanes / set_transforms are given (a program that has run the autotuner once keeps
                its choice); 0 leaves the engine's defaults
    steps       evaluations of a pass

Calls:

    step        one independent evaluation from host positions (Engine.compute): energies, forces, strain
    resident    the same with positions and forces on the device (Engine.launch_resident)
    md          a stretch of molecular dynamics: `steps` evaluations of moving positions with the dipole predictor and
                a kept pair list, host positions and forces (Engine.compute)
    device      the same stretch through the host package's device path: float4 positions, 64-bit fixed-point forces,
                the caller's stream (Engine.launch_device)
    batch       many independent boxes in one call (Engine.compute_batch)
    force_grad  an evaluation and the gradient of the force-matching loss with respect to every parameter (the backward
                direction; Engine.force_matching_grad), of one system or of a batch
    field       the field of given charges and dipoles at every atom (Engine.field): one application of the operator
"""

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent


def _package():
    """The package directory pgm-md_b200 under its import name."""
    name = "pgm_md_b200"
    if name not in sys.modules:
        path = ROOT / "pgm-md_b200"
        spec = importlib.util.spec_from_file_location(name, path / "__init__.py", submodule_search_locations=[str(path)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


def _case(name, call, system, molecules, precision="mixed", tol=1e-5, skin=0.0, lanes=0, transforms=0, systems=1, steps=1):
    c = dict(call=call, system=system, molecules=molecules, systems=systems, precision=precision, tol=tol, skin=skin,
             lanes=lanes, transforms=transforms, steps=steps)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: one evaluation of a small box from host memory (test boxes, small solutes, Monte Carlo),
        # where launches and latency count
        _case("water216-step", "step", "water", 216, tol=1e-6),
        # a small general cell in double precision, as used for checks and crystal work; an odd atom count
        _case("triclinic31-step-fp64", "step", "triclinic", 31, precision="fp64", tol=1e-8),
        # an ordinary box of a size that is a multiple of nothing, untuned engine
        _case("water1371-step", "step", "water", 1371),
        # the headline: one independent evaluation of the 8550-atom liquid, resident on the device, with the choices
        # that the autotuner makes there; and the same in double precision
        _case("dmp450-resident", "resident", "dimethylphenol", 450, lanes=16, transforms=4),
        _case("dmp450-resident-fp64", "resident", "dimethylphenol", 450, precision="fp64", lanes=16),
        # molecular dynamics of that liquid driven from host memory: predictor, kept pair list
        _case("dmp450-md", "md", "dimethylphenol", 450, skin=0.15, lanes=16, steps=8),
        # molecular dynamics of 4096 waters through the device path, as OpenMM's CUDA platform drives it
        _case("water4096-device", "device", "water", 4096, skin=0.15, steps=8),
        # the operator alone (one direct and one reciprocal field pass with its list)
        _case("dmp450-field-fp64", "field", "dimethylphenol", 450, precision="fp64"),
        # a large box
        _case("water32768-step", "step", "water", 32768, lanes=16),
        # many small boxes of 8..512 waters in one call
        _case("water-batch1024", "batch", "water", 512, systems=1024, lanes=16),
        # parameter fitting: the force-matching gradient of the 8550-atom liquid in double precision, and of 256 boxes
        # of 64 waters at once
        _case("dmp450-force-grad-fp64", "force_grad", "dimethylphenol", 450, precision="fp64", tol=1e-8),
        _case("water64x256-force-grad", "force_grad", "water", 64, systems=256, tol=1e-8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["step", "step", "resident", "md", "device", "batch", "force_grad", "field"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    lanes = rng.choice([0, 16, 32])
    transforms = rng.choice([0, 0, 3, 4])   # (where the grid or the precision does not allow one the engine takes 0)
    tol = rng.choice([1e-4, 1e-5, 1e-6])
    if call == "batch":
        return _case(None, call, "water", _log_int(rng, 8, 512), precision, tol, lanes=lanes,
                     systems=_log_int(rng, 2, 256))
    if call == "force_grad":
        if rng.random() < 0.5:
            return _case(None, call, "water", _log_int(rng, 16, 200), precision, 1e-8, systems=_log_int(rng, 2, 128))
        return _case(None, call, rng.choice(["water", "dimethylphenol"]), _log_int(rng, 30, 450), precision, 1e-8)
    system = rng.choice(["water", "water", "dimethylphenol", "triclinic"])
    top = {"water": 16384 if precision == "mixed" else 4096, "dimethylphenol": 800, "triclinic": 60}[system]
    molecules = _log_int(rng, {"water": 24, "dimethylphenol": 20, "triclinic": 8}[system], top)
    if call in ("md", "device"):
        return _case(None, call, system, min(molecules, 4096), precision, tol, skin=0.15, lanes=lanes,
                     transforms=transforms, steps=rng.choice([4, 6, 8]))
    return _case(None, call, system, molecules, precision, tol, skin=rng.choice([0.0, 0.0, 0.15]), lanes=lanes,
                 transforms=transforms)


# ------------------------------------------------------------------------------------------------ inputs

def _water(P, molecules, seed, tol, lattice=None):
    L = (molecules / 0.0334) ** (1.0 / 3.0)
    K = max(6, P.systems.fft_size(L / 1.0))
    return P.systems.waters(molecules, L, seed=seed, grid=(K, K, K), cutoff=min(9.0, L / 2.0), tol=tol, lattice=lattice)


def _dimethylphenol(P, molecules, seed, tol):
    """The C8H10O liquid of systems.dimethylphenol8550 with any number of molecules at its density: the parameters of
    that system's molecules, rigid molecules on a jittered lattice with random orientations."""
    S0 = P.systems.dimethylphenol8550(seed=seed, tol=tol)
    if molecules == 450:
        return S0
    rng = np.random.default_rng(seed + 1)
    L = 44.5 * (molecules / 450.0) ** (1.0 / 3.0)
    m = int(math.ceil(round((molecules * 512.0 / 450.0) ** (1.0 / 3.0), 9)))
    g = (np.arange(m) + 0.5) * (L / m)
    X, Y, Z = np.meshgrid(g, g, g, indexing="ij")
    sites = np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)[:molecules]
    sites = sites + rng.uniform(-0.2, 0.2, size=sites.shape)
    template = P.systems.dimethylphenol_template()[0]
    na, nb = len(template), len(S0.cov_atom) // 450
    R = P.systems.random_rotations(rng, molecules)
    pos = (np.einsum("mij,aj->mai", R, template) + sites[:, None, :]).reshape(-1, 3)
    base = np.repeat(na * np.arange(molecules), nb)
    K = max(6, P.systems.fft_size(L * 48.0 / 44.5))
    return P.systems.System(
        name="dimethylphenol", pos=pos * 0.1, box=np.eye(3) * L * 0.1, q=np.tile(S0.q[:na], molecules),
        radius=np.tile(S0.radius[:na], molecules), alpha=np.tile(S0.alpha[:na], molecules),
        cov_atom=base + np.tile(S0.cov_atom[:nb], molecules), cov_partner=base + np.tile(S0.cov_partner[:nb], molecules),
        cov_strength=np.tile(S0.cov_strength[:nb], molecules), cutoff=min(0.9, L * 0.05), beta=3.5, grid=(K, K, K),
        order=6, tol=tol)


def _system(P, case, seed):
    if case["system"] == "water":
        return _water(P, case["molecules"], 1000 + seed, case["tol"])
    if case["system"] == "dimethylphenol":
        return _dimethylphenol(P, case["molecules"], 8550 + seed, case["tol"])
    return P.systems.tiny_triclinic(nmol=case["molecules"], seed=7 + seed)


def _boxes(P, case, seed):
    """The boxes of a batch: molecule counts over the range for "batch", all alike for the gradients' training set."""
    if case["call"] == "batch":   # (the same counts for every seed)
        counts = np.random.default_rng(77).integers(8, case["molecules"] + 1, size=case["systems"])
    else:
        counts = np.full(case["systems"], case["molecules"])
    return [_water(P, int(m), 100003 * (seed + 1) + k, case["tol"]) for k, m in enumerate(counts)]


def _inputs(P, case, seed):
    """The host inputs of a case, made from the seed alone."""
    rng = np.random.default_rng(4242 + seed)
    batched = case["systems"] > 1
    systems = _boxes(P, case, seed) if batched else [_system(P, case, seed)]
    d = {"systems": systems, "pos": np.concatenate([s.pos for s in systems]), "boxes": np.stack([s.box for s in systems])}
    n = len(d["pos"])
    if case["call"] in ("md", "device"):
        # smooth motion: amplitude 0.01 nm, 100 steps a period, a phase per coordinate
        phase = rng.uniform(0, 2 * np.pi, d["pos"].shape)
        d["trajectory"] = [d["pos"] + 0.01 * np.sin(2 * np.pi * t / 100 + phase) for t in range(case["steps"])]
    if case["call"] == "force_grad":   # target forces of the magnitude that the systems' own have
        d["target"] = rng.normal(0.0, 1000.0, (n, 3))
    if case["call"] == "field":
        d["q"], d["d"] = systems[0].q.copy(), rng.normal(0.0, 0.01, (n, 3))
    return d


def _settings(P, case, S):
    gradient = case["call"] == "force_grad"
    return P.Settings(cutoff=S.cutoff, beta=S.beta, grid=S.grid, order=S.order, tol=case["tol"], max_iter=300,
                      peek=0.0 if gradient else 0.65, predictor=2 if case["call"] in ("md", "device") else 0,
                      ke=P.systems.KE_DEFAULT, skin=case["skin"],
                      precision=P.MIXED if case["precision"] == "mixed" else P.FP64)


FIXED_SCALE = float(1 << 32)


def prepare(case, seed):
    P = _package()
    st = _inputs(P, case, seed)
    systems = st["systems"]
    eng = P.Engine(_settings(P, case, systems[0]))
    if case["systems"] > 1:
        eng.set_systems(systems)
    else:
        eng.set_system(systems[0])
    if case["lanes"]:
        eng.set_pair_lanes(case["lanes"])
    if case["transforms"]:
        eng.set_transforms(case["transforms"])
    st.update(call=case["call"], engine=eng, batched=case["systems"] > 1, box=systems[0].box)
    if case["call"] == "resident":
        st["device_pos"] = torch.from_numpy(st["pos"]).cuda()
        st["device_forces"] = torch.zeros_like(st["device_pos"])
    if case["call"] == "device":
        q = systems[0].q[:, None]
        st["posq"] = [torch.from_numpy(np.concatenate([p, q], axis=1).astype(np.float32)).cuda()
                      for p in st["trajectory"]]
        st["fixed"] = torch.zeros((3, (len(q) + 31) // 32 * 32), dtype=torch.int64, device="cuda")
    return st


# ------------------------------------------------------------------------------------------------ a pass

def _terms(t):
    return np.array([t.direct, t.reciprocal, t.self, t.background, t.polarization])


def run(st):
    eng, call, box = st["engine"], st["call"], st["box"]
    if call == "step":
        r = eng.compute(st["pos"], box)
        return {"terms": _terms(r.terms), "forces": r.forces, "strain": r.strain}
    if call == "resident":
        stream = torch.cuda.current_stream().cuda_stream
        ok = False
        while not ok:   # (a pair list that outgrew its capacity: the evaluation is repeated)
            eng.launch_resident(st["device_pos"].data_ptr(), box, True, st["device_forces"].data_ptr(), stream)
            eng.wait_device(stream)
            ok, terms = eng.finish_device()
        return {"terms": _terms(terms), "forces": st["device_forces"], "strain": eng.strain_derivative()}
    if call == "md":
        eng.reset_history()
        out = [eng.compute(p, box) for p in st["trajectory"]]
        return {"terms": np.stack([_terms(r.terms) for r in out]), "forces": np.stack([r.forces for r in out])}
    if call == "device":
        stream = torch.cuda.current_stream().cuda_stream
        eng.reset_history()
        fixed, n = st["fixed"], len(st["pos"])
        terms, forces = [], []
        for posq in st["posq"]:
            ok = False
            while not ok:
                fixed.zero_()
                eng.launch_device(posq.data_ptr(), box, True, fixed.data_ptr(), fixed.shape[1], FIXED_SCALE, stream)
                eng.wait_device(stream)
                ok, t = eng.finish_device()
            terms.append(_terms(t))
            forces.append(fixed[:, :n].double() / FIXED_SCALE)
        return {"terms": np.stack(terms), "forces": forces}
    if call == "batch":
        r = eng.compute_batch(st["pos"], st["boxes"])
        return {"terms": r["energies"][:, :5], "forces": r["forces"], "strain": r["strain"]}
    if call == "force_grad":
        if st["batched"]:
            r = eng.compute_batch(st["pos"], st["boxes"])
            forces, terms = r["forces"], r["energies"][:, :5]
        else:
            r = eng.compute(st["pos"], box)
            forces, terms = r.forces, _terms(r.terms)
        loss, g, _ = eng.force_matching_grad(st["target"], tol=eng.settings.tol)
        return {"terms": terms, "forces": forces, "loss": loss, "q": g["q"], "radius": g["radius"], "alpha": g["alpha"],
                "strength": g["cov_strength"]}
    return {"field": eng.field(st["pos"], box, st["q"], st["d"])}


# ------------------------------------------------------------------------------------------------ work and tolerance

def _shape(case):
    """(atoms, pairs within the cutoff, grid points) of a case, from its densities."""
    atoms = pairs = points = 0
    for k in range(case["systems"]):
        m = case["molecules"]
        if case["call"] == "batch":   # the mean of the range
            m = (8 + m) / 2
        if case["system"] == "water":
            n, vol, rc = 3 * m, m / 33.4, min(0.9, 0.05 * (m / 0.0334) ** (1 / 3))
            grid = max(6.0, 10.0 * vol ** (1 / 3)) ** 3
        elif case["system"] == "dimethylphenol":
            n, vol = 19 * m, m / 450 * 4.45 ** 3
            rc, grid = min(0.9, 0.5 * vol ** (1 / 3)), 48.0 ** 3 * m / 450
        else:
            n, vol, rc, grid = 3 * m, 2.0 * 1.9 * 1.8, 0.85, 48.0 ** 3
        atoms, points = atoms + n, points + grid
        pairs += n * (n / vol) * 4.0 / 3.0 * math.pi * rc ** 3 / 2
    return int(atoms), int(pairs), int(points)


def work(case):
    n, pairs, points = _shape(case)
    # the inputs once (positions, three parameters an atom, a dipole entry for most atoms) and the outputs once
    per_atom = {"step": 24 + 24 + 16 + 24, "resident": 24 + 24 + 16 + 24, "batch": 24 + 24 + 16 + 24, "md": 24 + 24,
                "device": 16 + 24, "force_grad": 24 + 24 + 16 + 24 + 24 + 32, "field": 24 + 8 + 24 + 24}[case["call"]]
    # one operator application: 30 operations a pair, 2 x 216 points an atom at 4, two real transforms
    apply = 30.0 * pairs + 2 * 216 * 4.0 * n + 5.0 * points * math.log2(max(points, 2))
    setup = 150.0 * pairs          # the radial kernels of every pair
    final = 120.0 * pairs + 216 * 24.0 * n
    iterations = {1e-4: 6, 1e-5: 9, 1e-6: 11, 1e-8: 15}[case["tol"]]
    if case["call"] == "field":
        flops = setup + apply
    elif case["call"] == "force_grad":
        flops = 3 * setup + (2 * iterations + 4) * apply + 3 * final
    else:
        flops = setup + (iterations + 2) * apply + final
    if case["call"] in ("md", "device"):   # a predicted step takes fewer iterations
        flops = case["steps"] * (setup + 5 * apply + final)
    return {"bytes": float(per_atom * n * case["steps"]), "flops": float(flops)}


def tolerance(case):
    # about four times what the engine shows against exact() over the cases (up to 1.7e-6 mixed, 1.7e-13 fp64; the
    # solver and the predictor carry the rounding of sums in another order through their iterations)
    if case["precision"] == "fp64":
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 7e-6, "max": 3e-4}


# ------------------------------------------------------------------------------------------------ exact values

SQRT_PI = math.sqrt(math.pi)


def _min_image(v, H):
    """Minimum image in reduced triclinic boxes H (3, 3) or one per row: c, then b, then a."""
    v = list(v.unbind(-1))
    for c in (2, 1, 0):
        k = torch.round(v[c].detach() / H[..., c, c].detach())
        for j in range(3):   # (the upper entries vanish, not so their derivatives)
            v[j] = v[j] - k * H[..., c, j]
    return torch.stack(v, -1)


def _moduli(K, p):
    """|sum_k M_p(k + 1) exp(2 pi i m k / K)|^2, zeros replaced by the mean of their neighbours."""
    def spline(n, u):
        if n == 2:
            return max(0.0, 1.0 - abs(u - 1.0))
        return (u * spline(n - 1, u) + (n - u) * spline(n - 1, u - 1.0)) / (n - 1)

    data = np.zeros(K)
    for k in range(min(p - 1, K)):
        data[k] = spline(p, k + 1.0)
    mod = np.abs(np.fft.fft(data)) ** 2
    return np.where(mod < 1e-7, 0.5 * (np.roll(mod, 1) + np.roll(mod, -1)), mod)


class _Exact:
    """The pGM energy (Gaussian charges, covalent and induced dipoles under PME) of systems given as numpy arrays, in
    double precision: the direct sum over all pairs within the cutoff, B-spline PME with torch's FFT, the induced
    dipoles by the engine's documented solver (Jacobi-preconditioned conjugate gradients with a tolerance, a predictor
    and a peek step) and every derivative by automatic differentiation."""

    def __init__(self, systems, st, dev):
        self.dev, self.st = dev, st
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)
        ti = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.int64, device=dev)
        counts = np.array([len(s.q) for s in systems])
        first = np.concatenate([[0], np.cumsum(counts)])
        self.n, self.nsys, self.first = int(first[-1]), len(systems), first
        self.sys = ti(np.repeat(np.arange(self.nsys), counts))
        self.q, self.R, self.al = (t(np.concatenate([getattr(s, k) for s in systems])) for k in ("q", "radius", "alpha"))
        self.c = t(np.concatenate([s.cov_strength for s in systems]))
        self.ca, self.cp = (ti(np.concatenate([getattr(s, k) + o for s, o in zip(systems, first)]))
                            for k in ("cov_atom", "cov_partner"))
        self.H = t(np.stack([s.box for s in systems]))
        self.beta = t([s.beta for s in systems])
        self.cut = [s.cutoff for s in systems]
        self.order = systems[0].order
        self.groups = []
        for K in sorted({tuple(s.grid) for s in systems}):
            of = [k for k, s in enumerate(systems) if tuple(s.grid) == K]
            atoms = ti(np.concatenate([np.arange(first[k], first[k + 1]) for k in of]))
            local = ti(np.repeat(np.arange(len(of)), counts[of]))
            mod = [t(_moduli(k, self.order)) for k in K]
            m = [torch.fft.fftfreq(k, 1.0 / k, dtype=torch.float64, device=dev) for k in K[:2]]
            m.append(torch.arange(K[2] // 2 + 1, dtype=torch.float64, device=dev))
            m = torch.stack(torch.meshgrid(*[torch.where(a == -k / 2, -a, a) for a, k in zip(m, K)], indexing="ij"), -1)
            w = torch.full(m.shape[:3], 2.0, dtype=torch.float64, device=dev)
            w[..., 0] = 1.0
            if K[2] % 2 == 0:
                w[..., K[2] // 2] = 1.0
            bb = mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :K[2] // 2 + 1]
            self.groups.append((K, ti(of), atoms, local, m, w, bb))

    # ---- geometry
    def place(self, pos):
        """Positions: the pair list and, for the solver, everything that depends on them."""
        self.pos = torch.as_tensor(pos, dtype=torch.float64, device=self.dev)
        I, J = [], []
        for k in range(self.nsys):
            a, b, H, rc2 = int(self.first[k]), int(self.first[k + 1]), self.H[k], self.cut[k] ** 2
            step = max(1, (1 << 27) // max(1, b - a))
            for r0 in range(a, b, step):
                r1 = min(b, r0 + step)
                x = _min_image(self.pos[r0:r1, None, :] - self.pos[None, r0:b, :], H)
                hit = (x * x).sum(-1) < rc2
                i, j = torch.nonzero(torch.triu(hit, 1), as_tuple=True)
                I.append(i + r0)
                J.append(j + r0)
        self.i, self.j = torch.cat(I), torch.cat(J)
        x = self.pairs(self.pos, self.H)
        ar = x.norm(dim=-1) / torch.sqrt(2 * (self.R[self.i] ** 2 + self.R[self.j] ** 2))
        order = torch.argsort((ar >= 1.0).to(torch.int8), stable=True)   # the pairs with a r < 1 first
        self.near = int((ar < 1.0).sum())
        self.i, self.j = self.i[order], self.j[order]

    def pairs(self, pos, H):
        return _min_image(pos[self.i] - pos[self.j], H[self.sys[self.i]] if self.nsys > 1 else H[0])

    @staticmethod
    def _series(a, r, nmax):
        s, c, out = (a * r) ** 2, 2 * a / SQRT_PI, []
        for k in range(nmax):
            term, total = torch.ones_like(s), torch.zeros_like(s)
            for m in range(22):
                total = total + term / (2 * m + 2 * k + 1)
                term = -term * s / (m + 1)
            out.append(c * total)
            c = c * 2 * a * a
        return out

    @staticmethod
    def _complement(a, r, nmax):
        c, out = 2 / SQRT_PI * a * torch.exp(-(a * r) ** 2), [torch.erfc(a * r) / r]
        for k in range(1, nmax):
            out.append(((2 * k - 1) * out[-1] + c) / (r * r))
            c = c * 2 * a * a
        return out

    def kernels(self, x, R, nmax):
        r = x.norm(dim=-1)
        a = 1 / torch.sqrt(2 * (R[self.i] ** 2 + R[self.j] ** 2))
        b = self.beta[self.sys[self.i]]
        n = self.near
        lo = [u - v for u, v in zip(self._series(a[:n], r[:n], nmax), self._series(b[:n], r[:n], nmax))]
        hi = [v - u for u, v in zip(self._complement(a[n:], r[n:], nmax), self._complement(b[n:], r[n:], nmax))]
        return [torch.cat(p) for p in zip(lo, hi)]

    def perm(self, pos, H, c):
        v = _min_image(pos[self.cp] - pos[self.ca], H[self.sys[self.ca]] if self.nsys > 1 else H[0])
        return torch.zeros_like(pos).index_add(0, self.ca, c[:, None] * v / v.norm(dim=-1, keepdim=True))

    # ---- reciprocal space
    def splines(self, group, pos, H):
        """Per atom of a group: grid points (n, p^3), weights theta (3, n, p), their derivatives, K recip (n, 3, 3)."""
        K, of, atoms, local = group[:4]
        p = self.order
        rec = torch.linalg.inv(H[of])[local]                    # rec[k, a]: d s_a / d r_k
        # the grid coordinate: its integer part is of the unstrained geometry
        s = torch.einsum("nk,nka->na", pos[atoms], rec)
        Kt = torch.tensor(K, dtype=torch.float64, device=self.dev)
        w = Kt * (s - torch.floor(s.detach()))
        base = torch.floor(w.detach())
        fr = w - base
        M = [torch.ones_like(fr)]
        for k in range(2, p + 1):
            prev = M
            get = lambda j: prev[j] if 0 <= j < k - 1 else torch.zeros_like(fr)
            M = [((fr + j) * get(j) + (k - fr - j) * get(j - 1)) / (k - 1) for j in range(k)]
        get = lambda j: prev[j] if 0 <= j < p - 1 else torch.zeros_like(fr)
        th = torch.stack(M, -1)                                  # (n, 3, p)
        dth = torch.stack([get(j) - get(j - 1) for j in range(p)], -1)
        g = torch.remainder(base.long()[..., None] - torch.arange(p, device=self.dev), Kt.long()[:, None])
        at = (((local[:, None] * K[0] + g[:, 0])[:, :, None, None] * K[1] + g[:, 1][:, None, :, None]) * K[2]
              + g[:, 2][:, None, None, :]).reshape(len(local), -1)
        return at, th, dth, Kt * rec

    @staticmethod
    def _outer(a, b, c):
        return (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(len(a), -1)

    def charge_grid(self, group, sp, q, d):
        K, of, atoms = group[:3]
        at, th, dth, Kr = sp
        e = torch.einsum("nk,nka->na", d[atoms], Kr)[..., None]
        t, u = th.unbind(1), dth.unbind(1)
        w = self._outer(q[atoms][:, None] * t[0] + e[:, 0] * u[0], t[1], t[2])
        w = w + self._outer(t[0], e[:, 1] * u[1], t[2]) + self._outer(t[0], t[1], e[:, 2] * u[2])
        grid = torch.zeros(len(of) * K[0] * K[1] * K[2], dtype=torch.float64, device=self.dev)
        return grid.index_add(0, at.reshape(-1), w.reshape(-1)).reshape(len(of), *K)

    def influence(self, group, H):
        of, m, bb = group[1], group[4], group[6]
        Hs = H[of]
        ms = torch.einsum("xyza,ska->sxyzk", m, torch.linalg.inv(Hs))
        m2 = (ms * ms).sum(-1)
        safe = torch.where(m2 > 0, m2, torch.ones_like(m2))
        V = torch.linalg.det(Hs)[:, None, None, None]
        g = torch.exp(-(math.pi ** 2) * safe / self.beta[of][:, None, None, None] ** 2) / (math.pi * V * safe) / bb
        return torch.where(m2 > 0, g, torch.zeros_like(g))

    def prepare_operator(self):
        with torch.no_grad():
            self.x = self.pairs(self.pos, self.H)
            self.G = self.kernels(self.x, self.R, 3)
            self.sp = [self.splines(g, self.pos, self.H) for g in self.groups]
            self.infl = [self.influence(g, self.H) for g in self.groups]

    def field(self, q, d):
        """Direct, reciprocal and self field of charges q and dipoles d."""
        i, j, x = self.i, self.j, self.x
        G1, G2 = self.G[1][:, None], self.G[2][:, None]
        E = 4 * self.beta[self.sys][:, None] ** 3 / (3 * SQRT_PI) * d
        E.index_add_(0, i, (q[j][:, None] * G1 + (d[j] * x).sum(-1, keepdim=True) * G2) * x - d[j] * G1)
        E.index_add_(0, j, (-q[i][:, None] * G1 + (d[i] * x).sum(-1, keepdim=True) * G2) * x - d[i] * G1)
        for group, sp, g in zip(self.groups, self.sp, self.infl):
            K, atoms = group[0], group[2]
            F = torch.fft.rfftn(self.charge_grid(group, sp, q, d), dim=(1, 2, 3))
            phi = torch.fft.irfftn(F * g, s=K, dim=(1, 2, 3)) * (K[0] * K[1] * K[2])
            at, th, dth, Kr = sp
            ph = phi.reshape(-1)[at]
            t, u = th.unbind(1), dth.unbind(1)
            f = torch.stack([(self._outer(*[u[b] if a == b else t[b] for b in range(3)]) * ph).sum(-1)
                             for a in range(3)], -1)
            E.index_add_(0, atoms, -torch.einsum("nka,na->nk", Kr, f))
        return E

    # ---- the solver
    def per_system(self, v):
        return torch.zeros(self.nsys, dtype=torch.float64, device=self.dev).index_add_(0, self.sys, v.sum(-1))

    def cg(self, b, x, tol, norm=None):
        """(alpha^-1 - T) x = b per system from the guess x; x and the residual."""
        al, zero, sys = self.al[:, None], torch.zeros_like(self.q), self.sys

        def worst(r):
            m = torch.zeros(self.nsys, dtype=torch.float64, device=self.dev)
            return m.scatter_reduce_(0, sys, (al * r).abs().amax(-1), "amax", include_self=True)

        norm = self.per_system((al * b).abs()) / (3 * torch.bincount(sys, minlength=self.nsys)) + 1e-300
        r = b - (x / al - self.field(zero, x))
        z = al * r
        p, rz = z.clone(), self.per_system(r * z)
        active = worst(r) / norm > tol
        for _ in range(300):
            if not bool(active.any()):
                break
            on = active[sys][:, None]
            Ap = p / al - self.field(zero, p)
            alph = rz / self.per_system(p * Ap).clamp_min(1e-300)
            x = torch.where(on, x + alph[sys][:, None] * p, x)
            rn = torch.where(on, r - alph[sys][:, None] * Ap, r)
            z = al * rn
            beta = self.per_system(z * (rn - r)) / rz.clamp_min(1e-300)
            p = z + beta[sys][:, None] * p
            r, rz = rn, self.per_system(rn * z)
            active = active & (worst(r) / norm > tol)
        return x, r

    def dipoles(self, history=()):
        with torch.no_grad():
            self.prepare_operator()
            b = self.field(self.q, self.perm(self.pos, self.H, self.c))
            h = history
            if self.st.predictor == 2 and len(h) >= 4:
                x = 4 * h[0] - 6 * h[1] + 4 * h[2] - h[3]
            elif self.st.predictor and len(h) >= 3:
                x = 3 * h[0] - 3 * h[1] + h[2]
            elif self.st.predictor and h:
                x = h[0].clone()
            else:
                x = self.al[:, None] * b
            x, r = self.cg(b, x, self.st.tol)
            return x + self.st.peek * self.al[:, None] * r

    # ---- energies and derivatives
    def energies(self, pos, H, mu, q, R, al, c):
        """(nsys, 5) direct, reciprocal, self, background, polarization."""
        d = self.perm(pos, H, c) + mu
        i, j, x = self.i, self.j, self.pairs(pos, H)
        G = self.kernels(x, R, 3)
        dix, djx, didj = (d[i] * x).sum(-1), (d[j] * x).sum(-1), (d[i] * d[j]).sum(-1)
        U = q[i] * q[j] * G[0] + (q[i] * djx - q[j] * dix + didj) * G[1] - dix * djx * G[2]
        zero = torch.zeros(self.nsys, dtype=torch.float64, device=self.dev)
        direct = zero.index_add(0, self.sys[i], U)
        recip = zero
        for group in self.groups:
            F = torch.fft.rfftn(self.charge_grid(group, self.splines(group, pos, H), q, d), dim=(1, 2, 3))
            e = 0.5 * (group[5] * self.influence(group, H) * (F.real ** 2 + F.imag ** 2)).sum((1, 2, 3))
            recip = recip.index_add(0, group[1], e)
        b = self.beta[self.sys]
        self_e = zero.index_add(0, self.sys, -b / SQRT_PI * q * q - 2 * b ** 3 / (3 * SQRT_PI) * (d * d).sum(-1))
        Q = zero.index_add(0, self.sys, q)
        background = -math.pi * Q * Q / (2 * torch.linalg.det(H) * self.beta ** 2)
        pol = zero.index_add(0, self.sys, (mu * mu).sum(-1) / (2 * al))
        return self.st.ke * torch.stack([direct, recip, self_e, background, pol], -1)

    def evaluate(self, mu, strain=True):
        pos = self.pos.clone().requires_grad_(True)
        eps = torch.zeros(self.nsys, 3, 3, dtype=torch.float64, device=self.dev, requires_grad=True)
        A = torch.eye(3, dtype=torch.float64, device=self.dev) + eps
        e = self.energies(torch.einsum("nab,nb->na", A[self.sys], pos), torch.einsum("sab,skb->ska", A, self.H), mu,
                          self.q, self.R, self.al, self.c)
        gp, ge = torch.autograd.grad(e.sum(), (pos, eps))
        return e.detach(), -gp, ge.reshape(self.nsys, 9)

    def force_matching(self, mu, target, tol):
        """The loss sum |F - target|^2 at the solved dipoles and its gradient: with G = dE/dmu = 0 defining mu,
        dL/dtheta = d/dtheta [L + u . G] at fixed mu and u, (d2E/dmu2) u = -dL/dmu."""
        target = torch.as_tensor(target, dtype=torch.float64, device=self.dev)
        leaves = [v.clone().requires_grad_(True) for v in (self.pos, mu, self.q, self.R, self.al, self.c)]
        pos, m, q, R, al, c = leaves
        e = self.energies(pos, self.H, m, q, R, al, c)
        gp, gm = torch.autograd.grad(e.sum(), (pos, m), create_graph=True)
        L = ((-gp - target) ** 2).sum()
        dLdm = torch.autograd.grad(L, m, retain_graph=True)[0]
        with torch.no_grad():
            u, _ = self.cg(-dLdm / self.st.ke, torch.zeros_like(mu), tol)
        g = torch.autograd.grad(L + (u * gm).sum(), (q, R, al, c))
        return float(L.detach()), [v.detach() for v in g], e.detach(), -gp.detach()


def exact(case, seed):
    if case["systems"] * case["molecules"] > 60000:
        return None   # (over 20 seconds)
    P = _package()
    inp = _inputs(P, case, seed)
    systems, call = inp["systems"], case["call"]
    X = _Exact(systems, _settings(P, case, systems[0]), torch.device("cuda" if torch.cuda.is_available() else "cpu"))
    if call in ("md", "device"):
        history, terms, forces = [], [], []
        for p in inp["trajectory"]:
            X.place(p.astype(np.float32).astype(np.float64) if call == "device" else p)
            mu = X.dipoles(history)
            history = [mu] + history[:3]
            e, f, _ = X.evaluate(mu)
            terms.append(e[0])
            forces.append(f)
        if call == "device":
            return {"terms": torch.stack(terms), "forces": [f.T.contiguous() for f in forces]}
        return {"terms": torch.stack(terms), "forces": torch.stack(forces)}
    X.place(inp["pos"])
    if call == "field":
        with torch.no_grad():
            X.prepare_operator()
            t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=X.dev)
            return {"field": X.field(t(inp["q"]), t(inp["d"]))}
    mu = X.dipoles()
    if call == "force_grad":
        loss, (gq, gR, ga, gc), e, f = X.force_matching(mu, inp["target"], case["tol"])
        return {"terms": e if case["systems"] > 1 else e[0], "forces": f, "loss": loss, "q": gq, "radius": gR,
                "alpha": ga, "strength": gc}
    e, f, s = X.evaluate(mu)
    if call == "batch":
        return {"terms": e, "forces": f, "strain": s}
    return {"terms": e[0], "forces": f, "strain": s[0]}
