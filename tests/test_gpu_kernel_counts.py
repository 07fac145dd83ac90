"""The kernels a run reports (include/caps_gpu_diag.h): every step's, also where steps that rescale the cell run outside the
graphs, and where every thermo row falls on such a step."""
from __future__ import annotations

import pytest

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator
from tests.fixtures import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("barostat,every,rows", [("none", 10, 20), ("berendsen", 10, 20), ("c-rescale", 10, 7), ("berendsen", 4, 20),
                                                 ("berendsen", 40, 20), ("mtk", 1, 20)])
def test_every_step_is_counted(barostat, every, rows):
    fx = load("ps_small")
    eo = EnergyOptions(cutoff=8.0, skin=2.0, electrostatics="pme", pme_order=5, precision="mixed")
    thermostat = "nose-hoover" if barostat == "mtk" else "bussi"
    common = dict(dt=1.0, steps=40, temperature=300.0, tau_t=100.0, seed=4, energy=eo)
    plain = Evaluator(fx.ff, eo)
    plain.run(fx.x, fx.cell, DynamicsOptions(thermostat=thermostat, thermo_every=40, **common))
    step = plain.step_kernels()
    ev = Evaluator(fx.ff, eo)
    ev.run(fx.x, fx.cell, DynamicsOptions(thermostat=thermostat, thermo_every=rows, barostat=barostat, barostat_every=every, tau_p=500.0, **common))
    # a step has a plain step's kernels, in a block of steps one less (the velocity factor is left to the next step's first
    # kernel), and one that rescales the cell two force evaluations; twenty more are the most that a row or a rescaling adds
    special = sum(1 for s in range(1, 41) if barostat != "none" and s % every == 0)
    assert 40 * (step - 1) <= ev.kernels_run() <= 40 * (step + 2) + (special + 40 // rows + 1) * (step + 20)
    ev.close(), plain.close()
