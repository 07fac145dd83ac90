"""A list build that ends in an error leaves no list: the next evaluation builds it again, and reports the error again where
its cause still holds. The causes are made on the host: more atoms over one grid column than the column sort takes, more
excluded pairs than a super-cluster's table takes, and a wait between the list kernel's stages whose limit is set to nothing."""
from __future__ import annotations

import numpy as np
import pytest

from caps_b200 import DeviceError, DynamicsOptions, EnergyOptions, Evaluator, ForceField

pytestmark = pytest.mark.gpu


def _field(n, **kw):
    return ForceField(type_index=np.zeros(n, int), charge=np.zeros(n), mass=np.full(n, 12.0), pair_eps=[[0.1]], pair_sigma=[[2.6]],
                      element=np.full(n, 6), **kw)


def _cube(m, a):
    x = (np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3) + 0.5) * a
    return x + np.random.default_rng(2).uniform(-0.2, 0.2, x.shape)


def _cell(edge):
    return np.concatenate([np.zeros(3), np.diag(edge).reshape(-1)])


def _options(precision):
    return EnergyOptions(cutoff=6.0, skin=1.0, coulomb=False, precision=precision)


@pytest.mark.parametrize("precision", ["double", "mixed"])
def test_a_column_too_long_is_refused_each_time(precision):
    x = _cube((6, 6, 140), 3.2)                    # 5,040 atoms over one corner of a cell of 4 x 4 columns
    cell = _cell([160.0, 160.0, 448.0])
    ev = Evaluator(_field(len(x)), _options(precision))
    for _ in range(2):
        with pytest.raises(ValueError, match="grid column"):
            ev.compute(x, cell)
    ev.close()


@pytest.mark.parametrize("precision", ["double", "mixed"])
def test_too_many_excluded_partners_are_refused_each_time(precision):
    x = _cube((4, 4, 4), 3.2)                      # one super-cluster, every atom excluded from every other: 4,032 records
    others = np.arange(64) + np.arange(1, 64)[:, None]
    ff = _field(64, excl_offset=63 * np.arange(65), excl_list=np.sort(others % 64, axis=0).T.reshape(-1).astype(np.uint32))
    ev = Evaluator(ff, _options(precision))
    for _ in range(2):
        with pytest.raises(ValueError, match="excluded partners"):
            ev.compute(x, _cell([12.8] * 3))
    ev.close()


@pytest.mark.parametrize("precision", ["double", "mixed"])
def test_a_wait_that_gives_up_is_reported_and_the_next_call_is_right(precision):
    x = _cube((14, 14, 14), 3.2)
    cell = _cell([14 * 3.2] * 3)
    moved = x + 2.0                                # past half the skin: a build
    fresh = Evaluator(_field(len(x)), _options(precision))
    _, ref = fresh.compute(moved, cell)
    ev = Evaluator(_field(len(x)), _options(precision))
    ev.compute(x, cell)
    polls = 2 ** 21
    ev.set_list_wait(0)
    for _ in range(2):
        with pytest.raises(DeviceError, match="gave up waiting"):
            ev.compute(moved, cell)
    with pytest.raises(DeviceError, match="gave up waiting"):   # inside a run: the first force evaluation
        ev.run(moved, cell, DynamicsOptions(dt=1.0, steps=20, thermostat="none", temperature=50.0, thermo_every=20, seed=1, energy=_options(precision)))
    ev.set_list_wait(polls)
    _, f = ev.compute(moved, cell)
    assert np.abs(f - ref).max() <= 1e-9 * np.abs(ref).max()
    ev.close(), fresh.close()
