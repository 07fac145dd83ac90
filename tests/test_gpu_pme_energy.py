"""Energy and virial of the PME solve (the z transform's kernel) over grid lengths of every radix mix, odd and even, and every
spline order, against the same sums in numpy: the reciprocal sum with its half spectrum and Nyquist planes, the real-space
sum and the self term of a charged gas."""
from __future__ import annotations

import math

import numpy as np
import pytest

from caps_b200 import EnergyOptions, Evaluator, ForceField
from tests.test_gpu_pme_lines import KC, RC, RTOL, _bspline

pytestmark = pytest.mark.gpu


def _beta():
    lo, hi = 0.0, 20.0 / RC
    for _ in range(100):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if math.erfc(mid * RC) > RTOL else (lo, mid)
    return 0.5 * (lo + hi)


def _sums(x, q, edge, K, order, beta):
    """Energy, virial (xx yy zz xy xz yz) and the sizes of their terms."""
    u = (x / edge - np.floor(x / edge)) * K
    fu = np.floor(u)
    th = [_bspline(u[:, d] - fu[:, d], order) for d in range(3)]
    at = [(fu[:, d].astype(int)[:, None] - order + 1 + np.arange(order)) % K[d] for d in range(3)]
    grid = np.zeros(K)
    np.add.at(grid, (at[0][:, :, None, None], at[1][:, None, :, None], at[2][:, None, None, :]),
              q[:, None, None, None] * th[0][:, :, None, None] * th[1][:, None, :, None] * th[2][:, None, None, :])
    mod, m, nyquist = [], [], []
    for d in range(3):
        b = np.abs(np.exp(2j * np.pi * np.outer(np.arange(K[d]), np.arange(order)) / K[d]) @ _bspline(np.zeros(1), order)[0]) ** 2
        bad = b < 1e-7
        b[bad] = (0.5 * (np.roll(b, 1) + np.roll(b, -1)))[bad]
        k = np.arange(K[d])
        shape = [1, 1, 1]
        shape[d] = K[d]
        mod.append(b.reshape(shape))
        m.append((np.where(k >= (K[d] + 1) // 2, k - K[d], k) / edge[d]).reshape(shape))
        nyquist.append((2 * k == K[d]).reshape(shape))
    m2 = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
    m2[0, 0, 0] = 1
    fac = (math.pi / beta) ** 2
    G = KC * np.exp(-fac * m2) / (math.pi * np.prod(edge) * m2 * mod[0] * mod[1] * mod[2])
    G[0, 0, 0] = 0
    e = 0.5 * G * np.abs(np.fft.fftn(grid)) ** 2
    ss = 2 * (1 + fac * m2) / m2
    w = []
    for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
        both_signs = (a != b) & (nyquist[a] | nyquist[b])   # the average over +- of a Nyquist component
        w.append(float((e * ((a == b) - ss * np.where(both_signs, 0.0, m[a] * m[b]))).sum()))
    energy, size, wsize = float(e.sum()), float(e.sum()), float((e * (3 + ss * m2)).sum())
    w = np.array(w)
    for s in np.ndindex(3, 3, 3):
        d = x[None] - x[:, None]
        d = d - np.round(d / edge) * edge + (np.array(s) - 1) * edge
        r = np.sqrt((d * d).sum(-1))
        ok = (r < RC) & (r > 1e-9)
        r = np.where(ok, r, 1.0)
        er = np.vectorize(math.erfc)(beta * r)
        v = np.where(ok, 0.5 * KC * np.outer(q, q) * er / r, 0.0)
        g = np.where(ok, 0.5 * KC * np.outer(q, q) * (er / r + 2 * beta / math.sqrt(math.pi) * np.exp(-(beta * r) ** 2)) / r ** 2, 0.0)
        energy, size = energy + float(v.sum()), size + float(np.abs(v).sum())
        w = w + np.einsum("ij,ija,ijb->ab", g, d, d)[[0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2]]
        wsize += float((np.abs(g) * r * r).sum())
    self_term = KC * beta / math.sqrt(math.pi) * float((q * q).sum())
    return energy - self_term, w, size + self_term, wsize


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("K,order", [((9, 10, 12), 4), ((16, 15, 7), 5), ((35, 21, 25), 3), ((32, 27, 49), 6), ((45, 14, 63), 8), ((40, 18, 70), 7)])
def test_energy_and_virial(K, order, precision):
    edge = np.array(K) * 1.0
    rng = np.random.default_rng(sum(K) + order)
    n = 66
    x = rng.uniform(0, 1, (n, 3)) * edge
    for _ in range(200):      # no two charges on each other
        d = x[None] - x[:, None]
        d -= np.round(d / edge) * edge
        r = np.sqrt((d * d).sum(-1)) + 9 * np.eye(n)
        if r.min() > 1.0:
            break
        near = np.unique(np.argwhere(r < 1.0)[:, 0])[1:]
        x[near] = rng.uniform(0, 1, (len(near), 3)) * edge
    q = np.where(np.arange(n) % 2 == 0, 0.4, -0.4)
    ff = ForceField(type_index=np.zeros(n, int), charge=q, mass=np.full(n, 12.0), pair_eps=[[0.0]], pair_sigma=[[1.0]], element=np.full(n, 6))
    energy, w, size, wsize = _sums(x, q, edge, K, order, _beta())
    ev = Evaluator(ff, EnergyOptions(cutoff=RC, skin=1.0, electrostatics="pme", ewald_rtol=RTOL, pme_spacing=1.0, pme_order=order, tail=False,
                                     precision=precision))
    t, _ = ev.compute(x, np.concatenate([np.zeros(3), np.diag(edge).reshape(-1)]))
    ev.close()
    # double: the real-space table, 5e-11 of a term; float: 24 bits in the charges, weights and transforms of a few passes
    tol = 1e-9 if precision == "double" else 3e-6
    assert abs(t["coulomb"] - energy) <= tol * size, (t["coulomb"], energy, size)
    assert np.abs(np.array(t["w"]) - w).max() <= tol * wsize, (t["w"], w, wsize)
