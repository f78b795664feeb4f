"""Sorted order after steps, on both sides of the rule that picks the reorder
(131,072 particles: place and state in one launch below, two launches from
there on): integer work, exact against numpy's stable sort of the oracle's
cell keys, and every particle's state moves with it."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P
from psb_project_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 255, 20000, 131071, 131072])
@pytest.mark.parametrize("method", [P.WCSPH, P.PCISPH])
def test_order_and_state_after_a_step(n, method):
    sc = P.dam_break((64, 64, 32), 0.02, (1.6, 1.4, 0.8), 0.04, method=method, dt=1e-4, seed=3)
    pos = P.scene_positions(sc)[:n]
    sc = sc.replace(n=n)
    rng = np.random.default_rng(n)
    vel = rng.normal(0, 1.0, (n, 3)).astype(np.float32)
    with P.Simulation(sc) as sim:
        sim.upload(pos[rng.permutation(n)], vel, vel)
        sim.step(2)
        before = sim.download()
        sim.build_neighbors()               # no upload pending: the whole state moves
        keys = oracle.cell_keys(sc, before["pos"].astype(np.float64))
        assert np.array_equal(sim.read_field(R.FIELD_SORTED_ID), oracle.sort_perm(keys))
        assert np.array_equal(sim.read_field(R.FIELD_SORTED_KEY), np.sort(keys))
        after = sim.download()
    for name in ("pos", "vel", "vel_half"):
        assert np.array_equal(before[name], after[name]), name
