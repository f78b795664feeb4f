"""Iso field with particles outside the particle grid, which the build clamps
into border cells, or with a NaN coordinate, and node grids that reach past
it: a particle counts at a node only where the node's own ring of cells holds
it, whatever nodes share its brick. Grids with a node a thread and with bricks
of nodes, both kinds of cell ranges. FP64 sums in another order than the
oracle's: test_surface.py's 1e-12."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,spacing", [((33, 29, 31), 0.0095), ((75, 73, 74), 0.005)])
@pytest.mark.parametrize("box", [(0.2, 0.18, 0.2), (3.0, 3.5, 3.3)])      # counting sort's ranges; radix sort's
@pytest.mark.parametrize("nan", [False, True])
def test_field_of_particles_outside_the_grid(dims, spacing, box, nan):
    sc = P.dam_break((12, 10, 8), 0.01, box, 0.02, seed=5, jitter=1e-3)
    pos = P.scene_positions(sc)
    rng = np.random.default_rng(6)
    lo, hi = -0.02, 0.22                                  # the small box's grid, one cell around it
    out = pos[::4]                                        # a quarter of them past one to three faces
    far = rng.uniform(0.0, 0.05, out.shape).astype(np.float32)
    side = rng.integers(0, 3, out.shape)
    out[:] = np.where(side == 1, np.float32(lo) - far, np.where(side == 2, np.float32(hi) + far, out))
    if nan:
        for axis in range(3):
            pos[5 + 40 * axis, axis] = np.nan
        pos[205] = np.nan
    g = P.iso_grid((-0.1, -0.09, -0.095), spacing, dims)
    with P.Simulation(sc) as sim:
        sim.upload(pos)
        iso = sim.iso_field(g)
        rho = sim.read_field(P.runtime.FIELD_DENSITY)
    og = oracle.iso_grid(list(g.origin), list(g.spacing), list(g.dims), g.scale)
    want = oracle.iso_field(sc, pos.astype(np.float64), rho.astype(np.float64), og)
    assert np.array_equal(np.isnan(iso), np.isnan(want)) and np.isnan(want).any() == nan
    fin = ~np.isnan(want)
    assert np.max(np.abs(iso[fin] - want[fin])) <= 1e-12 * np.max(np.abs(want[fin]))
