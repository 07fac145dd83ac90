"""The PME transforms over grid lengths of every radix mix (one to three passes, odd line counts, lengths whose pairs of
lines leave one over) and every spline order, against the same sums in numpy: forces of a charged gas whose only
interaction is the reciprocal one with its real-space part."""
from __future__ import annotations

import math

import numpy as np
import pytest

from caps_b200 import EnergyOptions, ForceField

pytestmark = pytest.mark.gpu

KC, RTOL, RC = 332.06371, 1e-5, 4.5


def _bspline(w, p):
    th = [1 - w, w]
    for k in range(3, p + 1):
        th = [((w + k - 1 - j) * (th[j - 1] if j >= 1 else 0) + (j + 1 - w) * (th[j] if j < k - 1 else 0)) / (k - 1) for j in range(k)]
    return np.stack(th, -1)


def _reference(x, q, edge, K, order, beta):
    """Reciprocal forces on the grid K, and the real-space sum, in double."""
    n = len(x)
    u = (x / edge - np.floor(x / edge)) * K
    fu = np.floor(u)
    th = [_bspline(u[:, d] - fu[:, d], order) for d in range(3)]
    lo = [_bspline(u[:, d] - fu[:, d], order - 1) for d in range(3)]
    dth = [np.pad(t, ((0, 0), (1, 0))) - np.pad(t, ((0, 0), (0, 1))) for t in lo]
    at = [(fu[:, d].astype(int)[:, None] - order + 1 + np.arange(order)) % K[d] for d in range(3)]
    ix = (at[0][:, :, None, None], at[1][:, None, :, None], at[2][:, None, None, :])
    grid = np.zeros(K)
    np.add.at(grid, ix, q[:, None, None, None] * th[0][:, :, None, None] * th[1][:, None, :, None] * th[2][:, None, None, :])
    mod, m = [], []
    for d in range(3):
        b = np.abs(np.exp(2j * np.pi * np.outer(np.arange(K[d]), np.arange(order)) / K[d]) @ _bspline(np.zeros(1), order)[0]) ** 2
        bad = b < 1e-7
        b[bad] = (0.5 * (np.roll(b, 1) + np.roll(b, -1)))[bad]
        mod.append(b)
        k = np.arange(K[d])
        m.append(np.where(k >= (K[d] + 1) // 2, k - K[d], k) / edge[d])
    m2 = m[0][:, None, None] ** 2 + m[1][None, :, None] ** 2 + m[2][None, None, :] ** 2
    m2[0, 0, 0] = 1
    G = KC * np.exp(-(np.pi / beta) ** 2 * m2) / (np.pi * np.prod(edge) * m2 * mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :])
    G[0, 0, 0] = 0
    phi = np.fft.ifftn(np.fft.fftn(grid) * G).real * grid.size
    f = np.zeros((n, 3))
    for d in range(3):
        w = [dth[k] if k == d else th[k] for k in range(3)]
        f[:, d] = -q * K[d] / edge[d] * np.einsum("nabc,na,nb,nc->n", phi[ix], *w)
    for s in np.ndindex(3, 3, 3):
        d = x[None] - x[:, None]
        d = d - np.round(d / edge) * edge + (np.array(s) - 1) * edge
        r = np.sqrt((d * d).sum(-1))
        ok = (r < RC) & (r > 1e-9)
        r = np.where(ok, r, 1.0)
        er = np.vectorize(math.erfc)(beta * r)
        g = np.where(ok, KC * np.outer(q, q) * (er / r + 2 * beta / math.sqrt(math.pi) * np.exp(-(beta * r) ** 2)) / r ** 2, 0.0)
        f -= (g[..., None] * d).sum(1)
    return f


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("K,order", [((9, 10, 12), 4), ((16, 15, 7), 5), ((35, 21, 25), 3), ((32, 27, 49), 6), ((45, 14, 63), 8), ((40, 18, 70), 7)])
def test_grid_lengths_and_orders(K, order, precision):
    from caps_b200 import Evaluator
    edge = np.array(K) * 1.0
    rng = np.random.default_rng(sum(K))
    n = 66
    x = rng.uniform(0, 1, (n, 3)) * edge
    q = np.where(np.arange(n) % 2 == 0, 0.4, -0.4)
    for _ in range(200):      # no two charges on each other
        d = x[None] - x[:, None]
        d -= np.round(d / edge) * edge
        r = np.sqrt((d * d).sum(-1)) + 9 * np.eye(n)
        if r.min() > 1.0:
            break
        near = np.unique(np.argwhere(r < 1.0)[:, 0])[1:]
        x[near] = rng.uniform(0, 1, (len(near), 3)) * edge
    ff = ForceField(type_index=np.zeros(n, int), charge=q, mass=np.full(n, 12.0), pair_eps=[[0.0]], pair_sigma=[[1.0]], element=np.full(n, 6))
    cell = np.concatenate([np.zeros(3), np.diag(edge).reshape(-1)])
    ev = Evaluator(ff, EnergyOptions(cutoff=RC, skin=1.0, electrostatics="pme", ewald_rtol=RTOL, pme_spacing=1.0, pme_order=order, tail=False,
                                     precision=precision))
    lo, hi = 0.0, 20.0 / RC
    for _ in range(100):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if math.erfc(mid * RC) > RTOL else (lo, mid)
    ref = _reference(x, q, edge, K, order, 0.5 * (lo + hi))
    # double: 1e-8 of the largest force (the engine interpolates the real-space term from a table, 1e-9); float: 24 bits in
    # the charges, weights and a few hundred grid values summed per atom, 1e-5
    for _ in range(2):        # the second evaluation spreads on the grid that the first one left
        _, f = ev.compute(x, cell)
        assert np.abs(f - ref).max() <= (1e-8 if precision == "double" else 1e-5) * np.abs(ref).max()
    ev.close()
