"""Batches whose cells are rescaled, often enough that their steps are launched directly and seldom enough that they are replayed
from a graph, against the same replicas run one by one: the mixed path's results are the same bits (without constraints,
whose virial is summed in double in no fixed order)."""
from __future__ import annotations

import numpy as np
import pytest

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator, run_batch
from tests.fixtures import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [(1, 1), (2, 3), (7, 7), (31, 5), (32, 32), (7, 40)])
def test_batch_with_rescaling_equals_single_runs(every):
    eo = EnergyOptions(cutoff=8.0, skin=2.0, electrostatics="pme", pme_order=4, precision="mixed")
    reps = [(load("ps_small"), dict(thermostat="bussi", barostat="c-rescale", barostat_every=every[0])),
            (load("ps_medium"), dict(thermostat="nose-hoover", barostat="berendsen", barostat_every=every[1]))]
    opts = [DynamicsOptions(dt=1.0, steps=50, thermo_every=10, temperature=400.0, tau_t=100.0, tau_p=500.0, seed=3, energy=eo, **kw) for _, kw in reps]
    single = []
    for (fx, _), o in zip(reps, opts):
        ev = Evaluator(fx.ff, eo)
        single.append(ev.run(fx.x, fx.cell, o))
        ev.close()
    evs = [Evaluator(fx.ff, eo) for fx, _ in reps]
    for _ in range(2):   # the second time on engines that hold the first run's graphs
        batch = run_batch(evs, [fx.x for fx, _ in reps], [fx.cell for fx, _ in reps], opts)
        for a, b in zip(single, batch):
            assert [r["pressure"] for r in a["thermo"]] == [r["pressure"] for r in b["thermo"]]
            assert all(np.array_equal(a[k], b[k]) for k in ("x", "v", "cell"))
    for (fx, _), o, ev, a in zip(reps, opts, evs, single):   # and a single run afterwards
        b = ev.run(fx.x, fx.cell, o)
        assert all(np.array_equal(a[k], b[k]) for k in ("x", "v", "cell"))
        ev.close()
