"""The work a user of this engine has it do, as cases that can be timed: single-point force evaluations
(Evaluator.compute, what a minimiser, a relaxation or a trajectory's re-scoring calls), molecular dynamics
(Evaluator.run) and replicas in lock step (run_batch), from a few hundred atoms to a few hundred thousand, in both
precisions.

Structures. Polystyrene cells come from the repository's relaxed ones (198 and 2,064 atoms with GAFF-style mixing, 32,000
atoms with geometric mixing) and a charged triclinic cell from its fixtures; Kremer-Grest chains start back and forth through
a cubic lattice, rigid SPC/E water as a proton-ordered cubic lattice, both at the liquid's density. Each is repeated along
the cell's edges to the size of the case.
Every copy and every seed gets its own thermal displacements and velocities, so no two copies or seeds are alike.

A program that asks for the mixed path gets 32-bit arithmetic, and keeps its results in 32 bits, as the trajectory formats
the engine writes do; results of the FP64 path are kept in 64 bits.
"""
from __future__ import annotations

import functools
import math
from pathlib import Path

import numpy as np
import torch

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator, ForceField, run_batch
from caps_b200.systems import kg_melt, polystyrene_melt, spce_water, tile

ROOT = Path(__file__).resolve().parents[1]
KB = 0.0019872041       # kcal/(mol K)
ACC = 4.184e-4          # (kcal/mol/Å)/(g/mol) -> Å/fs^2
TAU = 48.888            # fs: the Kremer-Grest time unit for sigma = 1 Å, eps = 1 kcal/mol, m = 1 g/mol
KCOUL = 332.06371

GOLDEN = {"ps198": "ps_small", "ps2064": "ps_medium", "tri1100": "lj_triclinic"}
BASE_ATOMS = {"ps198": 198, "ps2064": 2064, "ps32k": 32000, "kg500": 500, "tri1100": 1100, "water24": 24}


# --- the cases ---------------------------------------------------------------------------------------------------
def _case(call, system, reps, **kw):
    c = {"call": call, "system": system, "na": reps[0], "nb": reps[1], "nc": reps[2], "precision": "mixed", "cutoff": 10.0,
         "electrostatics": "pme", "order": 4, "spacing": 1.0, "frames": 1, "steps": 0, "dt": 1.0, "thermostat": "bussi",
         "temperature": 300.0, "constraints": "none", "barostat": "none", "respa": 1, "thermo_every": 100, "replicas": ""}
    c.update(kw)
    return c


def listed():
    cases = [
        # a minimiser's call on a small cell with the default damped shifted force: latency and launches
        ("point 594 dsf", _case("compute", "ps198", (3, 1, 1), electrostatics="dsf")),
        # the parity path's evaluation of the 32k-atom melt (r_c 12 Å): a minimisation or an FP64 reference
        ("point 32k double", _case("compute", "ps32k", (1, 1, 1), precision="double", cutoff=12.0)),
        # re-scoring a trajectory: frames far apart, so that each builds its own list
        ("rescore 4 x 33k", _case("compute", "ps2064", (4, 2, 2), frames=4, order=5)),
        # the default run on the cell size of the reference's own scaling benchmark (about 600 atoms)
        ("md 594 dsf", _case("run", "ps198", (3, 1, 1), electrostatics="dsf", steps=200)),
        # coarse-grained Langevin on the FP64 path: 5,000 beads
        ("md kg 5000 double", _case("run", "kg500", (5, 2, 1), precision="double", electrostatics="none", steps=200, dt=0.01 * TAU,
                                    thermostat="langevin", temperature=1.0 / KB)),
        # a small box of rigid water, 2 fs, one replica of a property run
        ("md water 3000", _case("run", "water24", (5, 5, 5), steps=200, dt=2.0, constraints="h-bonds", spacing=1.2)),
        # a melt with the default PME order, constraints and pressure coupling, cells of unequal edges
        ("md npt 6192 shake", _case("run", "ps2064", (3, 1, 1), order=5, steps=100, dt=2.0, constraints="h-bonds",
                                    barostat="c-rescale", thermo_every=20)),
        # the 32k-atom melt in production: constraints, Nose-Hoover, PME
        ("md 32k nose-hoover", _case("run", "ps32k", (1, 1, 1), cutoff=12.0, steps=200, thermostat="nose-hoover", temperature=500.0,
                                     constraints="h-bonds")),
        # the same melt on the FP64 path without constraints
        ("md 32k double", _case("run", "ps32k", (1, 1, 1), precision="double", cutoff=12.0, steps=40, dt=0.5, temperature=500.0)),
        # replicas of uneven size in lock step (a cooling ladder's rung)
        ("batch 6 replicas", _case("batch", "ps2064", (1, 1, 1), steps=100, thermostat="langevin", temperature=400.0,
                                   replicas="1x1x1,2x1x1,3x1x1,2x2x1,3x2x1,2x2x2")),
        # a large melt with r-RESPA (PME outer) and stochastic cell rescaling
        ("md npt 128k respa", _case("run", "ps32k", (2, 2, 1), cutoff=12.0, steps=40, respa=2, barostat="c-rescale", temperature=500.0)),
        # 304,704 atoms of rigid water, 2 fs
        ("md water 305k", _case("run", "water24", (23, 23, 24), steps=40, dt=2.0, constraints="h-bonds", spacing=1.2)),
    ]
    return [dict(c, name=n) for n, c in cases]


def _reps(rng, most):
    """Repeats along three edges with a product spread over the logarithm of 1 .. most."""
    target = math.exp(rng.uniform(0.0, math.log(most + 0.999)))
    a = rng.randint(1, max(1, int(round(target ** 0.5))))
    b = rng.randint(1, max(1, int((target / a) ** 0.5)))
    c = max(1, int(target / (a * b)))
    r = [a, b, c]
    rng.shuffle(r)
    return tuple(r)


def _steps(rng, atoms, cost):
    """Steps of a run whose atom-steps stay under those of the largest listed case."""
    return max(10, min(rng.randint(60, 200), int(8.0e6 / (cost * atoms))))


def draw(rng):
    kind = rng.choice(["ps198", "ps2064", "ps2064", "ps32k", "kg500", "tri1100", "water24", "water24", "batch"])
    precision = rng.choice(["mixed", "mixed", "double"])
    cost = 2.5 if precision == "double" else 1.0
    if kind == "batch":
        return _case("batch", "ps2064", (1, 1, 1), steps=rng.randint(40, 100), thermostat=rng.choice(["langevin", "bussi", "nose-hoover"]),
                     temperature=float(rng.randint(150, 500)), replicas=",".join("%dx%dx%d" % _reps(rng, 6) for _ in range(rng.randint(2, 6))))
    if kind == "water24":
        m = math.exp(rng.uniform(math.log(4), math.log(20)))
        reps = tuple(max(4, int(round(m * rng.uniform(0.85, 1.15)))) for _ in range(3))
        n = 24 * reps[0] * reps[1] * reps[2]
        return _case("run", kind, reps, steps=_steps(rng, n, 1.0), dt=rng.choice([1.0, 2.0]), constraints="h-bonds",
                     spacing=rng.choice([1.0, 1.2]), order=rng.choice([4, 5]), thermostat=rng.choice(["bussi", "nose-hoover"]))
    if kind == "kg500":
        reps = _reps(rng, 40)
        n = 500 * reps[0] * reps[1] * reps[2]
        return _case("run", kind, reps, precision=precision, electrostatics="none", steps=_steps(rng, n, cost), dt=0.01 * TAU,
                     thermostat=rng.choice(["langevin", "nose-hoover"]), temperature=1.0 / KB)
    if kind == "tri1100":
        return _case("compute", kind, _reps(rng, 12), precision=precision, cutoff=rng.choice([8.0, 9.0, 10.0]),
                     electrostatics=rng.choice(["pme", "dsf"]), order=rng.choice([4, 5, 6]), frames=rng.randint(1, 3))
    reps = _reps(rng, {"ps198": 14, "ps2064": 14, "ps32k": 3}[kind])
    n = BASE_ATOMS[kind] * reps[0] * reps[1] * reps[2]
    el = rng.choice(["pme", "pme", "dsf"])
    cut = rng.choice([9.0, 10.0, 12.0])
    if rng.random() < 0.4:
        return _case("compute", kind, reps, precision=precision, cutoff=cut, electrostatics=el, order=rng.choice([4, 5]), frames=rng.randint(1, 3))
    cons = rng.choice(["none", "h-bonds"]) if precision == "mixed" else "none"
    return _case("run", kind, reps, precision=precision, cutoff=cut, electrostatics=el, order=rng.choice([4, 5]), steps=_steps(rng, n, 2 * cost),
                 thermostat=rng.choice(["bussi", "nose-hoover", "langevin"]), temperature=float(rng.randint(250, 500)), constraints=cons,
                 dt=1.0 if cons == "h-bonds" else 0.5)


# --- structures --------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _base(system):
    """(force field, x, cell) of one periodic cell."""
    if system == "ps32k":
        z = np.load(ROOT / "caps_b200" / "data" / "ps32k_start.npz")
        ff, _, _ = polystyrene_melt(40, 50, 1.04, seed=1, grow=False)
        return ff, z["x"].astype(np.float64), z["cell"].astype(np.float64)
    if system == "water24":
        # the cubic cell of eight rigid molecules with ordered protons: oxygens on a diamond lattice, every molecule's two
        # O-H bonds along two of its four O-O directions, so that each O-O contact has one proton
        ff, _, cell = spce_water(8, 0.997, seed=1)
        L = cell[3]
        fcc = np.array([[0, 0, 0], [0, 2, 2], [2, 0, 2], [2, 2, 0]], float) / 4.0
        up = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], float) / math.sqrt(3.0)
        x = []
        for f in fcc:      # sublattice A gives its protons towards two of its neighbours on B, B its own along the other two
            for o, d in ((f, (up[0], up[1])), (f + 0.25, (-up[2], -up[3]))):
                x += [o * L, o * L + d[0], o * L + d[1]]
        return ff, np.array(x), cell
    if system == "kg500":
        # ten chains of fifty beads laid back and forth through a simple cubic lattice at the melt's density
        ff, _, _ = kg_melt(10, 50, 0.85, seed=1)
        a = 0.85 ** (-1.0 / 3.0)
        path, y0 = [], list(range(10))
        for z in range(5):
            for k, y in enumerate(y0):
                path += [(c, y, z) for c in (range(10) if k % 2 == 0 else range(9, -1, -1))]
            y0 = y0[::-1]
        return ff, np.array(path, float) * a, np.array([0, 0, 0, 10 * a, 0, 0, 0, 10 * a, 0, 0, 0, 5 * a])
    z = np.load(ROOT / "tests" / "golden" / (GOLDEN[system] + ".npz"))
    return ForceField.from_arrays({k[3:]: z[k] for k in z.files if k.startswith("ff_")}), z["x"], z["cell"]


@functools.lru_cache(maxsize=4)
def _system(system, reps):
    ff, x, cell = _base(system)
    if reps == (1, 1, 1):
        return ff, np.asarray(x, np.float64).reshape(-1, 3), np.asarray(cell, np.float64).reshape(12)
    return tile(ff, x, cell, reps)


def _displaced(system, x, rng):
    """The structure with thermal displacements of its own: rigid ones for water, whose bonds have a fixed length."""
    if system != "water24":
        return x + rng.normal(0.0, 0.02, x.shape)
    m = x.reshape(-1, 3, 3)
    o = m[:, :1]
    w = rng.normal(0.0, 0.12, (len(m), 1, 3))       # small rotation vectors
    a = np.linalg.norm(w, axis=2, keepdims=True)
    k = w / a
    d = m - o
    d = d * np.cos(a) + np.cross(np.broadcast_to(k, d.shape), d) * np.sin(a) + k * (k * d).sum(2, keepdims=True) * (1 - np.cos(a))
    return (o + rng.normal(0.0, 0.06, o.shape) + d).reshape(-1, 3)


def _velocities(ff, temperature, rng):
    v = rng.normal(0.0, 1.0, (ff.natoms, 3)) * np.sqrt(KB * temperature * ACC / ff.mass)[:, None]
    return v - (ff.mass[:, None] * v).sum(0) / ff.mass.sum()


def _energy(case):
    if case["system"] == "kg500":
        return EnergyOptions(cutoff=2.0 ** (1 / 6), skin=0.4, coulomb=False, tail=False, precision=case["precision"])
    return EnergyOptions(cutoff=case["cutoff"], skin=2.0, electrostatics=case["electrostatics"], pme_spacing=case["spacing"],
                         pme_order=case["order"], precision=case["precision"])


def _dynamics(case, seed):
    return DynamicsOptions(dt=case["dt"], steps=case["steps"], temperature=case["temperature"], thermostat=case["thermostat"],
                           tau_t=2 * TAU if case["system"] == "kg500" else 100.0, barostat=case["barostat"], constraints=case["constraints"],
                           respa=case["respa"], respa_split="pme" if case["respa"] > 1 else "bonded", thermo_every=case["thermo_every"],
                           seed=seed, energy=_energy(case))


def _replicas(case):
    if case["call"] != "batch":
        return [(case["na"], case["nb"], case["nc"])]
    return [tuple(int(v) for v in r.split("x")) for r in case["replicas"].split(",")]


# --- a pass ------------------------------------------------------------------------------------------------------
def _inputs(case, seed):
    """Per replica (force field, cell, frames of positions, velocities)."""
    rng = np.random.default_rng(seed)
    out = []
    for reps in _replicas(case):
        ff, x, cell = _system(case["system"], reps)
        frames = []
        for k in range(case["frames"]):
            y = _displaced(case["system"], x, rng)
            if k:   # a later frame of a trajectory: the melt has drifted by several Å
                y = y + rng.uniform(-4.0, 4.0, 3)
            frames.append(np.ascontiguousarray(y))
        out.append((ff, cell, frames, _velocities(ff, case["temperature"], rng)))
    return out


def prepare(case, seed):
    """The engine(s) of the case's system and the structures to compute or to run from."""
    inputs = _inputs(case, seed)
    return {"case": case, "evaluators": [Evaluator(i[0], _energy(case)) for i in inputs], "inputs": inputs,
            "options": [_dynamics(case, 1 + r) for r in range(len(inputs))]}


TERMS = ("bond", "angle", "dihedral", "improper", "vdw", "coulomb", "virial", "total")
ROW = ("time_ps", "temperature", "kinetic", "potential", "total", "conserved", "pressure", "density")


def _held(case, a):
    return np.asarray(a, dtype=np.float64 if case["precision"] == "double" else np.float32)


def _run_result(case, r):
    return {"x": _held(case, r["x"]), "v": _held(case, r["v"]), "cell": _held(case, r["cell"]),
            "thermo": _held(case, [[row[k] for k in ROW] for row in r["thermo"]])}


def run(state):
    case, evs, inputs, opts = state["case"], state["evaluators"], state["inputs"], state["options"]
    if case["call"] == "compute":
        _, cell, frames, _ = inputs[0]
        got = [evs[0].compute(x, cell) for x in frames]
        out = {k: _held(case, [t[k] for t, _ in got]) for k in TERMS}
        out["w"] = _held(case, [t["w"] for t, _ in got])
        out["forces"] = _held(case, [f for _, f in got])
        return out
    if case["call"] == "run":
        ff, cell, frames, v = inputs[0]
        return _run_result(case, evs[0].run(frames[0], cell, opts[0], v=v))
    got = run_batch(evs, [i[2][0] for i in inputs], [i[1] for i in inputs], opts, vs=[i[3] for i in inputs])
    return [_run_result(case, r) for r in got]


def work(case):
    """Each input read and each output written once; the pairs inside the cut-off (59 operations each), the PME spread,
    transforms and gather and the bonded terms of every force evaluation."""
    size = {"double": 8, "mixed": 4}[case["precision"]]
    evals = case["frames"] if case["call"] == "compute" else case["steps"] + 1
    byts = flops = 0.0
    for reps in _replicas(case):
        ff, _, cell = _base(case["system"])
        m = reps[0] * reps[1] * reps[2]
        n = ff.natoms * m
        vol = abs(float(np.linalg.det(np.asarray(cell[3:]).reshape(3, 3)))) * m
        rc = 2.0 ** (1 / 6) if case["system"] == "kg500" else case["cutoff"]
        pairs = 0.5 * n * (4.0 / 3.0 * math.pi * rc ** 3 * n / vol)
        one = 59.0 * pairs
        if case["electrostatics"] == "pme":
            grid = vol / case["spacing"] ** 3
            one += n * case["order"] ** 3 * 10.0 + 2 * 2.5 * grid * math.log2(max(grid, 2.0))
        terms = m * (30.0 * len(ff.bond_ij) + 60.0 * len(ff.angle_ijk) + 120.0 * (len(ff.dihedral_ijkl) + len(ff.improper_ijkl)) +
                     30.0 * len(ff.pair14_ij) + 40.0 * len(ff.fene_ij))
        flops += evals * (one + terms + (60.0 * n if case["call"] != "compute" else 0.0))
        topology = m * 4.0 * (2 * ff.natoms + len(ff.excl_list) + ff.bond_ij.size + ff.angle_ijk.size + ff.dihedral_ijkl.size +
                              ff.improper_ijkl.size + ff.pair14_ij.size)
        state = 3.0 * n * (8 + size) * (2 if case["call"] != "compute" else case["frames"])
        byts += topology + state
    return {"bytes": byts, "flops": flops}


# --- the same evaluations in plain 64-bit torch --------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _bspline(w, p):
    """The p cardinal B-spline weights at fractional offset w [n], weight j for grid point floor(u) - p + 1 + j."""
    th = [1 - w, w]
    for k in range(3, p + 1):
        new = []
        for j in range(k):       # M_k at w + (k - 1 - j), from M_{k-1}
            y = w + (k - 1 - j)
            left = th[j - 1] if j >= 1 else 0.0     # M_{k-1}(y)
            right = th[j] if j < k - 1 else 0.0     # M_{k-1}(y - 1)
            new.append((y * left + (k - y) * right) / (k - 1))
        th = new
    return torch.stack(th, -1)


def _good_size(n):
    while True:
        k = n
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        if k == 1:
            return n
        n += 1


def _reciprocal(x, q, h, beta, order, spacing, strain):
    """Smooth PME: half the influence function times |structure factor|^2; m and the volume follow the strain."""
    dev = x.device
    K = [_good_size(max(order + 1, int(math.ceil(float(torch.linalg.norm(h[d])) / spacing)))) for d in range(3)]
    hi = torch.linalg.inv(h)                       # s = x hi, rows of h the cell's edges
    s = x @ hi
    grid = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=dev)
    th, base = [], []
    for d in range(3):
        u = (s[:, d] - torch.floor(s[:, d].detach())) * K[d]
        fu = torch.floor(u.detach())
        th.append(_bspline(u - fu, order))
        base.append((fu.long()[:, None] - order + 1 + torch.arange(order, device=dev)[None]) % K[d])
    w = q[:, None, None, None] * th[0][:, :, None, None] * th[1][:, None, :, None] * th[2][:, None, None, :]
    idx = (base[0][:, :, None, None] * K[1] + base[1][:, None, :, None]) * K[2] + base[2][:, None, None, :]
    grid = grid.index_add(0, idx.reshape(-1), w.reshape(-1)).reshape(K)
    S2 = torch.fft.fftn(grid).abs().square()
    mod = []
    for d in range(3):
        w0 = _bspline(torch.zeros(1, dtype=torch.float64), order)[0]          # M_p at the integers
        m = torch.arange(K[d], dtype=torch.float64)[:, None] * torch.arange(order, dtype=torch.float64)[None] * (2 * math.pi / K[d])
        b = (w0 * torch.cos(m)).sum(1).square() + (w0 * torch.sin(m)).sum(1).square()
        for k in range(K[d]):
            if b[k] < 1e-7:
                b[k] = 0.5 * (b[(k - 1) % K[d]] + b[(k + 1) % K[d]])
        mod.append(b.to(dev))
    bm = mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :]
    vol = torch.linalg.det(h @ strain).abs()
    his = torch.linalg.inv(h @ strain)
    fac = math.pi ** 2 / beta ** 2
    ms = []
    for d in range(3):
        m = torch.arange(K[d], dtype=torch.float64, device=dev)
        ms.append(torch.where(m >= (K[d] + 1) // 2, m - K[d], m))
    # an even grid's Nyquist index stands for both signs: the mean over them
    G = 0.0
    for sg in range(8):
        mm = []
        for d in range(3):
            m = ms[d].clone()
            if K[d] % 2 == 0 and (sg >> d) & 1:
                m[K[d] // 2] = -m[K[d] // 2]
            mm.append(m)
        mv = [mm[0][:, None, None] * his[r, 0] + mm[1][None, :, None] * his[r, 1] + mm[2][None, None, :] * his[r, 2] for r in range(3)]
        m2 = mv[0] * mv[0] + mv[1] * mv[1] + mv[2] * mv[2]
        m2 = m2 + torch.nn.functional.one_hot(torch.zeros(1, dtype=torch.long, device=dev), m2.numel()).reshape(m2.shape)
        g = KCOUL * torch.exp(-fac * m2) / (math.pi * vol * m2 * bm)
        mask = torch.ones_like(m2)
        mask[0, 0, 0] = 0
        G = G + g * mask / 8
    return 0.5 * (G * S2).sum()


def _erfc_as(x):
    """Abramowitz & Stegun 7.1.26, which defines the shifted-force constants."""
    t = 1 / (1 + 0.3275911 * x)
    return t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) * math.exp(-x * x)


def _one_exact(case, ff, cell, x):
    dev = _dev()
    f64 = dict(dtype=torch.float64, device=dev)
    n = ff.natoms
    X = torch.tensor(x, **f64)
    h = torch.tensor(np.asarray(cell[3:]).reshape(3, 3), **f64)
    hi = torch.linalg.inv(h)
    q = torch.tensor(ff.charge, **f64)
    ty = torch.tensor(ff.type_index, device=dev).long()
    eps, sig = torch.tensor(ff.pair_eps, **f64), torch.tensor(ff.pair_sigma, **f64)
    kg = case["system"] == "kg500"
    rc = ff.model_cutoff if ff.model_cutoff > 0 else case["cutoff"]
    coul, pme = not kg, not kg and case["electrostatics"] == "pme"
    tail = not kg and not ff.lj_shift
    kappa = 0.2
    if pme:
        lo, hi_ = 0.0, 20.0 / rc
        for _ in range(100):
            mid = 0.5 * (lo + hi_)
            lo, hi_ = (mid, hi_) if math.erfc(mid * rc) > 1e-5 else (lo, mid)
        kappa = 0.5 * (lo + hi_)
    ec = _erfc_as(kappa * rc)
    e0, f0 = ec / rc, ec / rc ** 2 + 2 * kappa / math.sqrt(math.pi) * math.exp(-(kappa * rc) ** 2) / rc
    vol = float(torch.linalg.det(h).abs())
    F = torch.zeros(n, 3, **f64)
    W = torch.zeros(3, 3, **f64)
    E = dict.fromkeys(("bond", "angle", "dihedral", "improper", "vdw", "coulomb"), 0.0)

    def nearest(i, j):
        d = X[j] - X[i]
        return d - torch.round(d @ hi) @ h

    def add(key, links, energy):
        """energy(separations) of links (i, j): forces and virial from its derivatives."""
        nonlocal F, W
        ds = [nearest(i, j).requires_grad_(True) for i, j in links]
        e = energy(*ds)
        E[key] += float(e.detach())
        for (i, j), d, g in zip(links, ds, torch.autograd.grad(e, ds)):
            F = F.index_add(0, j, -g).index_add(0, i, g)
            W = W - d.detach().T @ g

    def idx(a, k):
        return torch.tensor(np.asarray(a, dtype=np.int64)[:, k], device=dev)

    def par(a, k):
        return torch.tensor(np.asarray(a)[:, k], **f64)

    if len(ff.bond_ij):
        k, r0 = par(ff.bond_k_r0, 0), par(ff.bond_k_r0, 1)
        add("bond", [(idx(ff.bond_ij, 0), idx(ff.bond_ij, 1))], lambda d: (k * (d.norm(dim=1) - r0) ** 2).sum())
    if len(ff.fene_ij):
        fk, fr0, fe, fs = (par(ff.fene_k_r0_eps_sigma, c) for c in range(4))

        def fene(d):
            r = d.norm(dim=1)
            s6 = (fs / r) ** 6
            core = torch.where(r < 1.122462048309373 * fs, 4 * fe * (s6 * s6 - s6) + fe, torch.zeros_like(r))
            return (-0.5 * fk * fr0 ** 2 * torch.log(1 - (r / fr0) ** 2) + core).sum()
        add("bond", [(idx(ff.fene_ij, 0), idx(ff.fene_ij, 1))], fene)
    if len(ff.angle_ijk):
        i, j, k = (idx(ff.angle_ijk, c) for c in range(3))
        kt, t0 = par(ff.angle_kt_theta0, 0), par(ff.angle_kt_theta0, 1)
        add("angle", [(j, i), (j, k)], lambda u, v: (kt * (torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1)) - t0) ** 2).sum())
    for key, quad, vd, nn in (("dihedral", ff.dihedral_ijkl, ff.dihedral_v_delta, ff.dihedral_n),
                              ("improper", ff.improper_ijkl, ff.improper_v_delta, ff.improper_n)):
        if not len(quad):
            continue
        i, j, k, l = (idx(quad, c) for c in range(4))
        v, de = par(vd, 0), par(vd, 1)
        mult = torch.tensor(np.asarray(nn, float), **f64)

        def torsion(b1, b2, b3):
            m, p = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
            phi = torch.atan2(b2.norm(dim=1) * (b1 * p).sum(1), (m * p).sum(1))
            return (v * (1 + torch.cos(mult * phi - de))).sum()
        add(key, [(i, j), (j, k), (k, l)], torsion)

    def lj(r2, e, s, shift):
        q6 = (s * s / r2) ** 3
        v = 4 * e * (q6 * q6 - q6)
        if shift:
            qc = (s / rc) ** 6
            v = v - 4 * e * (qc * qc - qc)
        return v
    if len(ff.pair14_ij):
        i, j = idx(ff.pair14_ij, 0), idx(ff.pair14_ij, 1)
        scale = torch.full((len(i),), float(ff.lj14), **f64) if ff.pair14_lj is None else torch.tensor(ff.pair14_lj, **f64)
        add("vdw", [(i, j)], lambda d: (scale * lj((d * d).sum(1), eps[ty[i], ty[j]], sig[ty[i], ty[j]], not tail)).sum())

    def screened(r, qq):
        e = torch.erfc(kappa * r) / r
        return qq * (e if pme else e - e0 + f0 * (r - rc))

    # excluded pairs: the damped sum holds them, the bare Coulomb term (1 - factor) comes off
    off, lst = np.asarray(ff.excl_offset, np.int64), np.asarray(ff.excl_list, np.int64)
    ei = np.repeat(np.arange(n), np.diff(off))
    if coul and len(lst):
        half = ei < lst
        a, b = ei[half], lst[half]
        fac = np.zeros(len(a))
        if len(ff.pair14_ij):
            p = np.sort(np.asarray(ff.pair14_ij, np.int64), axis=1)
            keys = p[:, 0] * n + p[:, 1]
            val = np.full(len(p), float(ff.coul14)) if ff.pair14_coul is None else np.asarray(ff.pair14_coul, float)
            order = np.argsort(keys)
            at = np.clip(np.searchsorted(keys[order], a * n + b), 0, len(keys) - 1)
            hit = keys[order][at] == a * n + b
            fac = np.where(hit, val[order][at], 0.0)
        i, j = torch.tensor(a, device=dev), torch.tensor(b, device=dev)
        fc = torch.tensor(fac, **f64)
        qq = KCOUL * q[i] * q[j]

        def excluded(d):
            r = d.norm(dim=1)
            e = qq * (fc / r - torch.erf(kappa * r) / r)
            if not pme:
                e = torch.where(r < rc, e + qq * (-e0 + f0 * (r - rc)), torch.zeros_like(r))
            return e.sum()
        add("coulomb", [(i, j)], excluded)
    # the pairs inside the cut-off: every ordered pair and image, half each, but the excluded ones at their nearest image
    frac = X @ hi
    fw = frac - torch.floor(frac)
    xw = fw @ h
    shift0 = -torch.floor(frac)
    width = [vol / float(torch.linalg.cross(h[(d + 1) % 3], h[(d + 2) % 3]).norm()) for d in range(3)]
    reach = [int(math.floor(rc / w)) + 1 for w in width]
    ekey = torch.tensor(np.sort(ei * n + lst), device=dev) if len(lst) else None
    images = torch.cartesian_prod(*[torch.arange(-r, r + 1, device=dev) for r in reach]).to(torch.float64)
    chunk = max(1, int(2.5e7 / n))
    for S in images:
        zero = bool((S == 0).all())
        Sh = S @ h
        # only atoms that can reach the image's cell
        ok_i, ok_j = torch.ones(n, dtype=torch.bool, device=dev), torch.ones(n, dtype=torch.bool, device=dev)
        for d in range(3):
            t = rc / width[d]
            ok_j &= (fw[:, d] + S[d] >= -t) & (fw[:, d] + S[d] <= 1 + t)
            ok_i &= (fw[:, d] - S[d] >= -t) & (fw[:, d] - S[d] <= 1 + t)
        I, J = torch.nonzero(ok_i)[:, 0], torch.nonzero(ok_j)[:, 0]
        for s0 in range(0, len(I), chunk):
            ic = I[s0:s0 + chunk]
            r2 = torch.zeros(len(ic), len(J), **f64)
            for c in range(3):
                r2 += ((xw[J, c] + Sh[c])[None] - xw[ic, c][:, None]) ** 2
            hit = torch.nonzero(r2 < rc * rc)
            del r2
            i, j = ic[hit[:, 0]], J[hit[:, 1]]
            keep = (i != j) if zero else torch.ones_like(i, dtype=torch.bool)
            if ekey is not None:
                key = i * n + j
                at = torch.searchsorted(ekey, key).clamp(max=len(ekey) - 1)
                near = -torch.round((frac[j] - frac[i]))           # the image of j nearest to i, in unwrapped coordinates
                mine = S[None] + shift0[j] - shift0[i]
                keep &= ~((ekey[at] == key) & (near == mine).all(1))
            i, j = i[keep], j[keep]
            d = (xw[j] + Sh - xw[i]).requires_grad_(True)
            e_lj = 0.5 * lj((d * d).sum(1), eps[ty[i], ty[j]], sig[ty[i], ty[j]], not tail).sum()
            e_q = 0.5 * screened(d.norm(dim=1), KCOUL * q[i] * q[j]).sum() if coul else torch.zeros((), **f64)
            g, = torch.autograd.grad(e_lj + e_q, d)
            E["vdw"] += float(e_lj.detach())
            E["coulomb"] += float(e_q.detach())
            F = F.index_add(0, j, -g).index_add(0, i, g)
            W = W - d.detach().T @ g
    q2, qt = float((q * q).sum()), float(q.sum())
    if pme:
        xx = X.clone().requires_grad_(True)
        strain = torch.eye(3, **f64).requires_grad_(True)
        e = _reciprocal(xx, q, h, kappa, case["order"], case["spacing"], strain)
        g, gs = torch.autograd.grad(e, [xx, strain])
        F = F - g
        W = W - gs
        E["coulomb"] += float(e.detach()) - KCOUL * kappa / math.sqrt(math.pi) * q2
        if abs(qt) > 1e-10:
            eb = -KCOUL * math.pi * qt * qt / (2 * vol * kappa ** 2)
            E["coulomb"] += eb
            W = W + eb * torch.eye(3, **f64)
    elif coul:
        E["coulomb"] -= (ec / (2 * rc) + f0 * rc / 2 + kappa / math.sqrt(math.pi)) * q2 * KCOUL
    W = 0.5 * (W + W.T)
    if tail:
        cnt = torch.bincount(ty, minlength=len(eps)).double()
        s6 = sig ** 6
        nn = cnt[:, None] * cnt[None]
        et = float((nn * 8 * math.pi * eps * (s6 * s6 / (9 * rc ** 9) - s6 / (3 * rc ** 3))).sum()) / vol
        wt = float((nn * 8 * math.pi * eps * (4 * s6 * s6 / (3 * rc ** 9) - 2 * s6 / rc ** 3)).sum()) / vol
        E["vdw"] += et
        W = W + wt / 3 * torch.eye(3, **f64)
    E["virial"] = float(W.diagonal().sum())
    E["total"] = sum(E[k] for k in TERMS[:6])
    E["w"] = [float(W[a, b]) for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    return E, F.cpu().numpy()


def exact(case, seed):
    """Single-point evaluations in 64 bits. Runs of many steps have no such value: a plain step takes seconds, and a
    trajectory is not a number that two roundings share."""
    if case["call"] != "compute" or sum(a * b * c for a, b, c in _replicas(case)) * BASE_ATOMS[case["system"]] > 40000:
        return None
    ff, cell, frames, _ = _inputs(case, seed)[0]
    got = [_one_exact(case, ff, cell, x) for x in frames]
    out = {k: np.array([e[k] for e, _ in got]) for k in TERMS}
    out["w"] = np.array([e["w"] for e, _ in got])
    out["forces"] = np.array([f for _, f in got])
    return out
