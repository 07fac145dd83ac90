"""The pair list and both pair kernels at every depth of work items, with damped Coulomb, in rectangular and triclinic cells and
with grid columns up to the longest that the column sort takes: energies, all six components of the virial and forces against
a direct sum in double, and the force-only kernels of plain steps through a short run from rest."""
from __future__ import annotations

import functools
import math

import numpy as np
import pytest

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator, ForceField

pytestmark = pytest.mark.gpu

RC, ALPHA, KC, ACC = 5.0, 0.25, 332.06371, 4.184e-4
EPS, SIG = np.array([[0.1, 0.15], [0.15, 0.2]]), np.array([[2.6, 2.7], [2.7, 2.9]])
A = 3.2
# sites along the three edges, and what each site's first, second and third step adds to the other directions
CELLS = {"cube": ((6, 6, 6), np.eye(3)), "tilted": ((8, 7, 10), np.array([[1, 0, 0], [0.3, 1, 0], [-0.25, 0.2, 1]])),
         "turned": ((7, 9, 8), np.array([[0.8, 0.6, 0], [-0.5, 0.85, 0.1], [0.2, -0.1, 1]])),
         "column of 2,240": ((4, 4, 140), np.eye(3)), "column of 4,000": ((4, 4, 250), np.eye(3))}


@functools.lru_cache(maxsize=None)
def _system(name):
    """Force field, positions, edges (rows), and the direct sum's energies, virial, forces and the sizes of their terms."""
    from scipy.spatial import cKDTree
    m, h = CELLS[name]
    rng = np.random.default_rng(len(name))
    sites = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    x = (sites + 0.5 + rng.uniform(-0.12, 0.12, sites.shape)) @ (A * h)
    n = len(x)
    q = rng.normal(0.0, 0.3, n)
    q -= q.mean()
    ff = ForceField(type_index=np.arange(n) % 2, charge=q, mass=np.full(n, 12.0), pair_eps=EPS, pair_sigma=SIG, element=np.full(n, 6))
    edges = np.array(m)[:, None] * A * h
    shifts = np.stack(np.meshgrid(*[[-1, 0, 1]] * 3, indexing="ij"), -1).reshape(-1, 3) @ edges   # every width is over twice the cut-off
    images = (x[None] + shifts[:, None]).reshape(-1, 3)
    near = cKDTree(images).query_ball_point(x, RC)
    i = np.repeat(np.arange(n), [len(k) for k in near])
    k = np.concatenate(near).astype(int)
    d = images[k] - x[i]
    r2 = (d * d).sum(1)
    keep = (r2 > 1e-9) & (r2 < RC * RC)
    i, j, d, r2 = i[keep], k[keep] % n, d[keep], r2[keep]
    r = np.sqrt(r2)
    e, s6 = EPS[i % 2, j % 2], SIG[i % 2, j % 2] ** 6
    r6, c6 = s6 / r2 ** 3, s6 / RC ** 6
    vdw = 4 * e * (r6 * r6 - r6 - c6 * c6 + c6)
    # the shift of the damped sum takes erfc from Abramowitz & Stegun 7.1.26, as the reference does
    t = 1 / (1 + 0.3275911 * ALPHA * RC)
    ex = math.exp(-(ALPHA * RC) ** 2)
    er = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) * ex
    f0 = er / RC ** 2 + 2 * ALPHA / math.sqrt(math.pi) * ex / RC
    erfc = np.array([math.erfc(ALPHA * v) for v in r])
    qq = KC * q[i] * q[j]
    coul = qq * (erfc / r - er / RC + f0 * (r - RC))
    g = 24 * e * (2 * r6 * r6 - r6) / r2 + qq * (erfc / r2 + 2 * ALPHA / math.sqrt(math.pi) * np.exp(-(ALPHA * r) ** 2) / r - f0) / r
    f = np.zeros((n, 3))
    np.add.at(f, i, -g[:, None] * d)
    w = 0.5 * np.einsum("k,ka,kb->ab", g, d, d)[[0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2]]
    self_term = (er / (2 * RC) + f0 * RC / 2 + ALPHA / math.sqrt(math.pi)) * (q * q).sum() * KC
    sizes = 0.5 * np.abs(vdw).sum(), 0.5 * np.abs(coul).sum() + self_term, 0.5 * (np.abs(g) * r2).sum()
    return ff, x, edges, 0.5 * vdw.sum(), 0.5 * coul.sum() - self_term, w, f, sizes


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("name,depth", [(c, None) for c in CELLS] + [("tilted", d) for d in (1, 2, 4, 8, 16, 24, 32)] + [("column of 4,000", 24)])
def test_against_direct_sum(name, depth, precision):
    ff, x, edges, vdw, coul, w, f, sizes = _system(name)
    cell = np.concatenate([np.zeros(3), edges.reshape(-1)])
    eo = EnergyOptions(cutoff=RC, skin=1.2, electrostatics="dsf", dsf_alpha=ALPHA, tail=False, precision=precision)
    ev = Evaluator(ff, eo)
    if depth:
        ev.pin_tuning([depth] + ev.tuning()[1:])
    # double: the table of the damped Coulomb term, 5e-11 of a term at most. float: 2^-24 in a separation, fourteen times that in
    # r^-14: 1e-6 of a pair's force, of which the largest here is some ten times an atom's, and less where many are summed
    tol = 1e-9 if precision == "double" else 3e-6
    t, force = ev.compute(x, cell)
    assert abs(t["vdw"] - vdw) <= tol * sizes[0] and abs(t["coulomb"] - coul) <= tol * sizes[1]
    assert np.abs(np.array(t["w"]) - w).max() <= tol * sizes[2]
    assert np.abs(force - f).max() <= 10 * tol * np.abs(f).max()
    # three steps of 0.001 fs from rest move an atom by 1e-9 A: v = 3 dt f / m, two thirds of it from the plain steps' kernels
    dt = 1e-3
    out = ev.run(x, cell, DynamicsOptions(dt=dt, steps=3, thermostat="none", thermo_every=3, temperature=0.0, seed=1, energy=eo), v=np.zeros_like(x))
    got = out["v"].reshape(-1, 3) * 12.0 / (3 * dt * ACC)
    assert np.abs(got - f).max() <= 10 * max(tol, 1e-8) * np.abs(f).max()
    ev.close()


@pytest.mark.parametrize("kind", ["a force cap that nothing reaches", "frozen pairs"])
@pytest.mark.parametrize("name", list(CELLS))
def test_fp64_rare_variants_against_direct_sum(name, kind):
    ff, x, edges, vdw, coul, w, f, sizes = _system(name)
    cell = np.concatenate([np.zeros(3), edges.reshape(-1)])
    ev = Evaluator(ff, EnergyOptions(cutoff=RC, skin=1.2, electrostatics="dsf", dsf_alpha=ALPHA, tail=False, precision="double",
                                     force_cap=1e6 if "cap" in kind else 0.0))
    if kind == "frozen pairs":
        ev.freeze_pairs(x, cell)
    t, force = ev.compute(x, cell)
    ev.close()
    assert abs(t["vdw"] - vdw) <= 1e-9 * sizes[0] and abs(t["coulomb"] - coul) <= 1e-9 * sizes[1]
    assert np.abs(np.array(t["w"]) - w).max() <= 1e-9 * sizes[2]
    assert np.abs(force - f).max() <= 1e-8 * np.abs(f).max()


def test_fp64_work_items_stop_at_sixteen_entries():
    """Deeper ones take a block per SM from the FP64 pair kernel (98,304 atoms: 429 us a launch at 24 entries, 339 at 16)."""
    m, a = 48, 2.2
    x = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    n = len(x)
    ff = ForceField(type_index=np.zeros(n, int), charge=np.zeros(n), mass=np.full(n, 12.0), pair_eps=[[0.1]], pair_sigma=[[2.0]],
                    element=np.full(n, 6))
    ev = Evaluator(ff, EnergyOptions(cutoff=12.0, skin=2.0, electrostatics="dsf", precision="double"))
    ev.compute(x, np.concatenate([np.zeros(3), np.diag([m * a] * 3).reshape(-1)]))
    assert ev.tuning()[0] == 16
    ev.close()
