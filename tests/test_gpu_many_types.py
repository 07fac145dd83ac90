"""Force fields of many atom types on the FP64 path, whose pair kernel keeps the table of type pairs in shared memory beside a
work item's atoms and the Ewald table: the most types that the engine takes, with Coulomb tables of 1,025 nodes and of some
thousands, at the engine's own depth of work items and at the deepest, against the same system with two types."""
from __future__ import annotations

import numpy as np
import pytest

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator, ForceField

pytestmark = pytest.mark.gpu


def _gas(nt):
    """600 sites of nt types, even ones of one kind and odd ones of another."""
    rng = np.random.default_rng(3)
    m, a = np.array([10, 10, 6]), 3.3
    x = (np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3) + rng.uniform(0.35, 0.65, (600, 3))) * a
    t = rng.integers(0, nt // 2 * 2, 600)
    t[:nt] = np.arange(nt)
    odd = np.arange(nt) % 2
    eps, sig = np.array([[0.1, 0.15], [0.15, 0.2]]), np.array([[2.6, 2.7], [2.7, 2.9]])
    pick = np.ix_(odd, odd)
    ff = ForceField(type_index=t, charge=np.where(np.arange(600) % 2 == 0, 0.3, -0.3), mass=np.full(600, 12.0), pair_eps=eps[pick],
                    pair_sigma=sig[pick], element=np.full(600, 6))
    two = ForceField(type_index=t % 2, charge=ff.charge, mass=ff.mass, pair_eps=eps, pair_sigma=sig, element=ff.element)
    return ff, two, x, np.concatenate([np.zeros(3), np.diag(m * a).reshape(-1)])


@pytest.mark.parametrize("cap", [0.0, 1e6])
@pytest.mark.parametrize("depth", [None, 32])
@pytest.mark.parametrize("alpha", [None, 0.3, 0.85, 1.0, 1.1, 1.3])   # 1,025 / 1,851 / 2,561 / 3,099 / 4,328 nodes
def test_many_types_equal_two(alpha, depth, cap):
    ff, two, x, cell = _gas(63)
    eo = EnergyOptions(cutoff=8.0, skin=1.5, coulomb=alpha is not None, electrostatics="dsf", dsf_alpha=alpha or 0.2, precision="double",
                       force_cap=cap)
    out = []
    for f in (ff, two):
        ev = Evaluator(f, eo)
        if depth:
            ev.pin_tuning([depth] + ev.tuning()[1:])
        t, force = ev.compute(x, cell)
        md = ev.run(x, cell, DynamicsOptions(dt=1.0, steps=2, thermostat="none", temperature=300.0, seed=5, thermo_every=2, energy=eo))
        out.append((t["total"], t["virial"], force, md["v"]))
        ev.close()
    # the same sums in another order: 1e-16 a term, some hundred terms an atom
    (ea, va, fa, xa), (eb, vb, fb, xb) = out
    assert abs(ea - eb) <= 1e-11 * abs(eb) and abs(va - vb) <= 1e-11 * max(abs(vb), abs(eb))
    assert np.abs(fa - fb).max() <= 1e-12 * np.abs(fb).max()
    assert np.abs(xa - xb).max() <= 1e-12 * np.abs(xb).max()
