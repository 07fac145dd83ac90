"""A batch queues its replicas' first evaluations one behind another. An engine that still has to choose its launch shapes does
so by timing evaluations: no other replica's kernel may run beside those (seen in the kernels' times and streams)."""
from __future__ import annotations

import json
import tempfile

import numpy as np
import pytest

from caps_b200 import DynamicsOptions, EnergyOptions, Evaluator, ForceField, run_batch

pytestmark = pytest.mark.gpu


def _gas(m):
    n, a = m ** 3, 3.6
    x = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    ff = ForceField(type_index=np.zeros(n, int), charge=np.where(np.arange(n) % 2 == 0, 0.1, -0.1), mass=np.full(n, 12.0),
                    pair_eps=[[0.1]], pair_sigma=[[3.0]], element=np.full(n, 6))
    return ff, x + np.random.default_rng(m).uniform(-0.1, 0.1, x.shape), np.concatenate([np.zeros(3), np.diag([m * a] * 3).reshape(-1)])


def _kernels(call):
    import torch
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    with tempfile.NamedTemporaryFile(suffix=".json") as tf:
        prof.export_chrome_trace(tf.name)
        trace = json.load(open(tf.name))
    ev = [e for e in trace["traceEvents"] if e.get("cat") == "kernel"]
    return sorted((e["ts"], e["ts"] + e["dur"], e["args"]["stream"]) for e in ev)


def test_shapes_are_timed_alone():
    ea = EnergyOptions(cutoff=24.0, skin=1.0, electrostatics="dsf", precision="double")   # some milliseconds an evaluation
    eb = EnergyOptions(cutoff=9.0, skin=1.0, electrostatics="pme", precision="double")
    (fa, xa, ca), (fb, xb, cb) = _gas(80), _gas(11)
    opts = [DynamicsOptions(dt=1.0, steps=2, thermostat="none", thermo_every=2, temperature=100.0, seed=2, energy=e) for e in (ea, eb)]
    a = Evaluator(fa, ea)
    for _ in range(2):                                 # the second time all but the small replica's engine is warm
        b = Evaluator(fb, eb)
        mine = {s for _, _, s in _kernels(lambda: a.compute(xa, ca))}
        ks = _kernels(lambda: run_batch([a, b], [xa, xb], [ca, cb], opts, vs=[np.zeros_like(xa), None]))
        b.close()
    a.close()
    timed = [k for k in ks if k[2] not in mine][:200]  # the small one's: 144 evaluations of some kernels each
    other = [k for k in ks if k[2] in mine]
    assert len(timed) == 200 and len(other) > 0
    beside = [k for k in timed for q in other if k[0] < q[1] and q[0] < k[1]]
    assert not beside, len(beside)
