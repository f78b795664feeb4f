"""Infinite and NaN coordinates in the neighbour build, which collects the
signs of |d|^2 - h^2: such a particle is clamped into a border cell and is
nobody's neighbour, nor its own, as in the reference's test by comparison.
(3e38 is finite: |d|^2 overflows, but particles that share it are neighbours.)
Alone in a quad of candidates and filling quads, with both kinds of cell
ranges. Counts are exact against the oracle."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P
from psb_project_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(0.3, 0.2, 0.25), (3.0, 3.5, 3.3)])      # counting sort's ranges; radix sort's
@pytest.mark.parametrize("every", [1, 2, 37])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3e38])
@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1, 2)])
def test_not_finite_is_no_neighbour(box, every, bad, axes):
    sc = P.dam_break((14, 6, 5), 0.01, box, 0.02, seed=2, jitter=2e-3, nbr_cap=512)
    pos = P.scene_positions(sc) - np.float32(0.015)       # up to the grid's corner, where the clamped ones go
    for a in axes:
        pos[::every, a] = bad
    counts, _ = oracle.neighbors(sc, pos.astype(np.float64))
    with P.Simulation(sc) as sim:
        sim.upload(pos)
        sim.build_neighbors()
        assert np.array_equal(sim.read_field(R.FIELD_NBR_COUNT), counts)
        assert sim.stats().nbr_total == counts.sum()
    assert np.isfinite(bad) or (counts[::every] == 0).all()
