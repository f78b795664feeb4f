"""The neighbour build's rows of candidates at their edges: lattices with
1 to ~100 candidates per row of cells (up to 32 a row the masks path, beyond
it the chunked one), clouds with both kinds in one warp, list capacities that
are not a multiple of four, both kinds of cell ranges. Counts are exact
against the oracle; the density over the lists has the parity suite's 1e-5."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P
from psb_project_b200 import runtime as R

pytestmark = pytest.mark.gpu


def check(sc, pos):
    counts, lists = oracle.neighbors(sc, pos.astype(np.float64))
    rho = oracle.density(sc, pos.astype(np.float64), counts, lists, clamp=True)
    with P.Simulation(sc) as sim:
        sim.upload(pos)
        sim.build_neighbors()
        assert np.array_equal(sim.read_field(R.FIELD_NBR_COUNT), counts)
        got = sim.read_field(R.FIELD_DENSITY_X).astype(np.float64)
        st = sim.stats()
        assert st.nbr_max == counts.max() and st.nbr_total == counts.sum()
    assert np.max(np.abs(got - rho) / rho) <= 1e-5


@pytest.mark.parametrize("box", [(0.3, 0.2, 0.25), (3.0, 3.5, 3.3)])      # counting sort's ranges; radix sort's
@pytest.mark.parametrize("per_cell", [0.3, 1, 4, 10, 12, 33])
def test_row_lengths(per_cell, box):
    h = 0.02
    s = h / per_cell ** (1 / 3)
    m = tuple(max(3, int(round(0.08 / s)) + k) for k in (1, 0, 2))
    sc = P.dam_break(m, s, box, h, seed=2, jitter=0.2 * s, nbr_cap=512)
    check(sc, P.scene_positions(sc) + np.float32(0.04))


@pytest.mark.parametrize("n", [31, 33, 700])
@pytest.mark.parametrize("cap", [128, 255, 510])
def test_crowded_and_sparse_rows_in_one_warp(n, cap):
    sc = P.dam_break((n, 1, 1), 0.01, (0.3, 0.2, 0.25), 0.02, seed=1, nbr_cap=cap).replace(n=n)
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.05, 0.15, (n, 3))
    pos[: n // 4] = [0.1, 0.1, 0.1] + rng.normal(0, 0.006, (n // 4, 3))
    pos = pos.astype(np.float32)
    if oracle.neighbors(sc.replace(nbr_cap=512), pos.astype(np.float64))[0].max() > cap:
        pytest.skip("the cloud's largest list exceeds this capacity")
    check(sc, pos)
