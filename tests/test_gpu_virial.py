"""All six components of the pair virial against a direct sum in numpy for ordered structures, whose pair forces have
components that are exactly zero: lattices, a displaced row of one, dimers along each axis away from the first atom of their
super-cluster."""
from __future__ import annotations

import numpy as np
import pytest

from caps_b200 import EnergyOptions, Evaluator, ForceField

pytestmark = pytest.mark.gpu

RC, EPS, SIG = 5.0, 0.2, 2.8


def _lattice(m=(6, 5, 7), a=3.0):
    x = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3) * a + 0.5
    return x, np.array(m) * a


def _structure(name):
    """Positions, edges, which atoms interact."""
    if name == "lattice":
        x, edge = _lattice()
        return x, edge, np.ones(len(x), bool)
    if name.startswith("row"):
        x, edge = _lattice()
        axis = "xyz".index(name[-1])
        k, l = [d for d in range(3) if d != axis]
        x[(x[:, k] == 6.5) & (x[:, l] == 6.5), axis] += 0.4
        return x, edge, np.ones(len(x), bool)
    axis = "xyz".index(name[-1])   # inert atoms below and above a dimer along the axis
    x = np.array([[1.0, 1, 1], [10, 4, 6], [10, 4, 6], [19, 19, 19]])
    x[2, axis] += 3.0
    return x, np.full(3, 20.0), np.array([False, True, True, False])


def _direct(x, edge, on):
    w, size, energy = np.zeros((3, 3)), 0.0, 0.0
    e = EPS * np.outer(on, on)
    for s in np.ndindex(3, 3, 3):   # every edge is longer than twice the cut-off
        d = x[None] - x[:, None] + (np.array(s) - 1) * edge
        r2 = (d * d).sum(-1)
        ok = (r2 < RC * RC) & (r2 > 0)
        r2 = np.where(ok, r2, 1.0)
        r6 = np.where(ok, (SIG * SIG / r2) ** 3, 0.0)
        c6 = (SIG / RC) ** 6
        energy += 0.5 * np.where(ok, 4 * e * (r6 * r6 - r6 - c6 * c6 + c6), 0.0).sum()
        g = 24 * e * (2 * r6 * r6 - r6) / r2
        w += 0.5 * np.einsum("ij,ija,ijb->ab", g, d, d)
        size += 0.5 * (np.abs(g) * np.where(ok, r2, 0.0)).sum()
    return w[[0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2]], size, energy


@pytest.mark.parametrize("kind", ["double", "double with a force cap", "mixed"])
@pytest.mark.parametrize("name", ["lattice", "row x", "row y", "row z", "dimer x", "dimer y", "dimer z"])
def test_virial_of_ordered_structures(name, kind):
    x, edge, on = _structure(name)
    n = len(x)
    ff = ForceField(type_index=(~on).astype(int), charge=np.zeros(n), mass=np.full(n, 12.0), pair_eps=[[EPS, 0.0], [0.0, 0.0]],
                    pair_sigma=[[SIG, SIG], [SIG, SIG]], element=np.full(n, 6))
    ev = Evaluator(ff, EnergyOptions(cutoff=RC, skin=1.0, coulomb=False, tail=False, precision=kind.split()[0],
                                     force_cap=1e6 if "cap" in kind else 0.0))
    t, _ = ev.compute(x, np.concatenate([np.zeros(3), np.diag(edge).reshape(-1)]))
    ev.close()
    ref, size, energy = _direct(x, edge, on)
    # double: sums of a force times a position of at most four times the cut-off, some hundred terms each; float: 2^-24 in the
    # separation, fourteen times that in r^-14, averaged over the pairs
    tol = 1e-12 if kind != "mixed" else 3e-6
    assert np.abs(np.array(t["w"]) - ref).max() <= tol * size, (t["w"], ref)
    assert abs(t["vdw"] - energy) <= tol * size, (t["vdw"], energy)


def test_mixed_sums_do_not_depend_on_how_pairs_are_grouped():
    """Every pair's energy and virial are rounded to fixed point on their own: the sums over all pairs equal, to the last
    unit, those of the same atoms with one pair of types interacting at a time, which parts the pairs of each work item."""
    rng = np.random.default_rng(7)
    x, edge = _lattice((7, 7, 7), 2.9)
    x = x + rng.uniform(-0.2, 0.2, x.shape)
    n, nt = len(x), 4
    types = rng.integers(0, nt, n)

    def sums(eps):
        ff = ForceField(type_index=types, charge=np.zeros(n), mass=np.full(n, 12.0), pair_eps=eps, pair_sigma=np.full((nt, nt), SIG),
                        element=np.full(n, 6))
        ev = Evaluator(ff, EnergyOptions(cutoff=RC, skin=1.0, coulomb=False, tail=False, precision="mixed"))
        t, _ = ev.compute(x, np.concatenate([np.zeros(3), np.diag(edge).reshape(-1)]))
        ev.close()
        return np.array(t["w"] + [t["vdw"]])

    parts = np.zeros(7)
    for a in range(nt):
        for b in range(a, nt):
            eps = np.zeros((nt, nt))
            eps[a, b] = eps[b, a] = EPS
            parts += sums(eps)
    assert np.array_equal(sums(np.full((nt, nt), EPS)), parts)
