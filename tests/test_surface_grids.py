"""Iso field and surface on node grids at the kernels' edges: dimensions that
are not a multiple of the bricks, spacings on both sides of half a cell and
beyond one, unequal spacings, grids that start outside the box and lie far
from the origin. The field and the mesh have the tolerances of
test_surface.py (FP64 sums in another order: 1e-12; float terms in the
reference profile: 1e-6; identical triangles of the GPU's own field)."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", ["config", "ref"])
@pytest.mark.parametrize("dims,spacing,origin", [
    ((2, 2, 2), 0.02, (0.02, 0.02, 0.02)),
    ((9, 8, 7), 0.01, (0.0, 0.0, 0.0)),
    ((75, 73, 74), 0.005, (-0.03, -0.02, -0.01)),        # enough nodes for bricks of them
    ((75, 73, 74), (0.005, 0.0101, 0.005), (-0.03, -0.2, -0.01)),      # but one spacing over half a cell
    ((33, 5, 17), (0.002, 0.02, 0.004), (0.01, 0.01, 0.01)),
    ((31, 41, 29), 0.004, (-0.05, -0.03, -0.04)),        # starts outside the box
    ((13, 12, 11), 0.026, (-0.1, -0.1, -0.1)),           # coarser than a cell
])
def test_ragged_grids_match_oracle(profile, dims, spacing, origin):
    if profile == "ref":
        sc = P.ref_scene((12, 10, 8), seed=5, jitter=2e-3)
        level = 4.0
    else:
        sc = P.dam_break((12, 10, 8), 0.01, (0.3, 0.25, 0.2), 0.02, seed=5, jitter=1e-3)
        level = 0.5
    pos = P.scene_positions(sc)
    g = P.iso_grid(origin, spacing, dims, scale=0.65)
    with P.Simulation(sc) as sim:
        sim.upload(pos)
        iso = sim.iso_field(g)
        vert, tri = sim.extract_surface(g, level)
        rho = sim.read_field(P.runtime.FIELD_DENSITY)
    og = oracle.iso_grid(list(g.origin), list(g.spacing), list(g.dims), g.scale)
    want = oracle.iso_field(sc, pos.astype(np.float64), rho.astype(np.float64), og)
    assert np.max(np.abs(iso - want)) <= (1e-6 if profile == "ref" else 1e-12) * np.max(np.abs(want))
    ov, ot = oracle.marching_cubes(og, iso, level)
    assert np.array_equal(tri, ot)
    if len(ov):
        assert np.max(np.abs(vert - ov)) <= 2 * np.spacing(np.float32(np.max(np.abs(ov))))
