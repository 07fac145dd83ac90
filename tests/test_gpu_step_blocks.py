"""Blocks of plain steps replayed as one graph (a run's steps between two thermo rows, eight at a time) against the same run
with a row every seven steps, which is too often for a block: every thermostat, with r-RESPA and with constraints, in both
precisions; and the total energy of a run without a thermostat against an absolute bound."""
from __future__ import annotations

import numpy as np
import pytest

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator
from tests.fixtures import load

pytestmark = pytest.mark.gpu

EXTRA = {"plain": {}, "respa": dict(respa=2, dt=1.0), "pme split": dict(respa=2, respa_split="pme", dt=1.0),
         "constraints": dict(constraints="h-bonds", dt=1.0)}


def _run(precision, rows, steps, **kw):
    fx = load("ps_small")
    eo = EnergyOptions(cutoff=8.0, skin=2.0, electrostatics="pme", pme_order=5, precision=precision)
    o = DynamicsOptions(**{**dict(dt=0.5, steps=steps, temperature=300.0, tau_t=100.0, seed=4, energy=eo, thermo_every=rows), **kw})
    ev = Evaluator(fx.ff, eo)
    out = ev.run(fx.x, fx.cell, o)
    ev.close()
    return out


# r-RESPA takes no Nose-Hoover chain and no Langevin thermostat
PAIRS = [(e, t) for e in EXTRA for t in ("none", "bussi") + (() if "respa" in EXTRA[e] else ("nose-hoover", "langevin"))]


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("extra,thermostat", PAIRS)
def test_blocks_equal_single_steps(extra, thermostat, precision):
    kw = dict(thermostat=thermostat, **EXTRA[extra])
    a, b = (_run(precision, rows, 40, **kw) for rows in (40, 7))
    # the two sum their forces in another order: 1e-15 of a force in double, 1e-6 of it in float, over 40 steps at most a
    # hundred times that of a velocity; SHAKE and RATTLE stop at 1e-8, which a sum's last bit can move by a sweep (1e-8 A a
    # step, 1e-5 of a velocity)
    tol = 1e-9 if precision == "double" and extra != "constraints" else 1e-4
    v, ref = np.asarray(a["v"]), np.asarray(b["v"])
    assert np.abs(v - ref).max() <= tol * np.sqrt(np.mean(ref ** 2)) * 10
    assert abs(a["thermo"][-1]["total"] - b["thermo"][-1]["total"]) <= tol * abs(b["thermo"][0]["kinetic"])


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("extra", ["plain", "respa", "pme split"])
def test_energy_without_thermostat_stays(extra, precision):
    # velocity Verlet's energy swings by (w dt)^2 / 8 of a mode's: 1 % for C-H bonds (11 fs) at 0.5 fs, at the inner step here;
    # 5 % of the kinetic energy is far above what all modes together show, and far below what a lost velocity costs
    out = _run(precision, 25, 200, thermostat="none", **EXTRA[extra])
    total = [r["total"] for r in out["thermo"]]
    assert max(total) - min(total) <= 0.05 * out["thermo"][0]["kinetic"]
