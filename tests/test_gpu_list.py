"""The list kernel and the work items' depth (caps_b200/csrc/list.cuh) against a direct sum in numpy: sizes around the
kernel's units (64-atom super-clusters, 256-thread blocks, columns of one and several super-clusters), a fresh list, a
kept one, a pruned one and a rebuilt one, in both precisions."""
from __future__ import annotations

import numpy as np
import pytest

from caps_b200 import EnergyOptions, ForceField

pytestmark = pytest.mark.gpu

RC, SKIN = 5.0, 1.5


def _gas(n, shape, seed):
    """n neutral Lennard-Jones sites on a jittered lattice in a box of the given edge ratios, chains of four excluded."""
    rng = np.random.default_rng(seed)
    edge = np.array(shape) * (n / 0.03 / np.prod(shape)) ** (1.0 / 3.0)
    m = np.maximum(1, np.round(edge / (edge.prod() / n) ** (1.0 / 3.0)).astype(int))
    while m.prod() < n:
        m[np.argmin(m / edge)] += 1
    sites = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)[:n]
    x = (sites + 0.5 + rng.uniform(-0.15, 0.15, (n, 3))) / m * edge
    off, lst = [0], []
    for i in range(n):
        lst += [j for j in range(i - i % 4, min(i - i % 4 + 4, n)) if j != i]
        off.append(len(lst))
    ff = ForceField(type_index=np.arange(n) % 2, charge=np.zeros(n), mass=np.full(n, 12.0), pair_eps=[[0.1, 0.15], [0.15, 0.2]],
                    pair_sigma=[[2.6, 2.7], [2.7, 2.9]], excl_offset=np.array(off), excl_list=np.array(lst, np.uint32), element=np.full(n, 6))
    return ff, x, np.concatenate([np.zeros(3), np.diag(edge).reshape(-1)])


def _direct(ff, x, cell):
    edge = np.array([cell[3], cell[7], cell[11]])
    n = len(x)
    excl = np.zeros((n, n), bool)
    for i in range(n):
        excl[i, ff.excl_list[ff.excl_offset[i]:ff.excl_offset[i + 1]]] = True
    e, s6 = ff.pair_eps[ff.type_index][:, ff.type_index], ff.pair_sigma[ff.type_index][:, ff.type_index] ** 6
    d0 = x[None] - x[:, None]
    near = np.round(d0 / edge)
    reach = np.ceil(RC / edge + 0.5).astype(int) - 1   # about the nearest image
    f, energy = np.zeros_like(x), 0.0
    for a in range(-reach[0], reach[0] + 1):
        for b in range(-reach[1], reach[1] + 1):
            for c in range(-reach[2], reach[2] + 1):
                img = np.array([a, b, c])
                d = d0 - near * edge + img * edge
                r2 = (d * d).sum(-1)
                ok = r2 < RC * RC
                if not img.any():
                    ok &= ~excl & ~np.eye(n, dtype=bool)
                r6 = np.where(ok, s6 / np.where(ok, r2, 1.0) ** 3, 0.0)
                energy += 0.5 * float((4 * e * (r6 * r6 - r6)).sum())
                g = np.where(ok, 24 * e * (2 * r6 * r6 - r6) / np.where(ok, r2, 1.0), 0.0)
                f -= (g[..., None] * d).sum(1)
    return energy, f


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("n,shape", [(2, (1, 1, 1)), (63, (1, 1, 1)), (65, (1, 1, 4)), (257, (3, 1, 1)), (511, (1, 2, 1)), (1537, (1, 1, 6))])
def test_list_stages_against_direct_sum(n, shape, precision):
    from caps_b200 import Evaluator
    ff, x, cell = _gas(n, shape, n)
    ev = Evaluator(ff, EnergyOptions(cutoff=RC, skin=SKIN, coulomb=False, tail=True, precision=precision))
    rng = np.random.default_rng(1)
    # forces of separations of some Å: 1e-12 in double; in float 3e-5 of the largest pair force (2^-24 in the separations
    # and the coefficients, amplified 13 times by r^-13 and summed over at most 60 neighbours of random sign)
    tol = 1e-12 if precision == "double" else 3e-5
    steps = [np.zeros(3), rng.uniform(-0.05, 0.05, (n, 3)),       # a fresh list, a kept one
             rng.uniform(-0.3, 0.3, (n, 3)),                      # past half the prune margin: pruned again
             np.array([7.0, -3.0, 11.0])]                         # past half the skin: rebuilt
    built, moved, pruned_at = [], [], x
    for move in steps:
        x = x + move
        moved.append(np.linalg.norm(x - pruned_at, axis=1).max())
        _, f = ev.compute(x, cell)
        _, ref = _direct(ff, x, cell)
        assert np.abs(f - ref).max() <= tol * max(1.0, np.abs(ref).max()), (n, precision)
        built.append(ev.list_counts())
    assert built[0][0] >= 1 and built[1][0] == built[0][0] and built[3][0] == built[2][0] + 1, built
    # half the prune margin of 0.8 Å: an atom past it since the first list's prune asks for another
    assert moved[1] < 0.4 and built[1][1] == built[0][1] and built[2][1] == built[1][1] + int(moved[2] > 0.4), (built, moved)
    ev.close()
