"""The two forms of the fluid's reaction on boundary particles (one warp each
up to 8,192 particles, one thread each above): the same terms in the same
order, so particles far from all others, added to cross the line, leave the
forces on the first ones the same to the bit."""
import numpy as np
import pytest

import psb_project_b200 as P

pytestmark = pytest.mark.gpu

H = 0.02


def forces(sc, fluid, pressure, solid):
    with P.Simulation(sc) as sim:
        sim.set_boundary(solid)
        sim.upload(fluid, pressure=pressure)
        sim.presolve(0)            # lists and density; the uploaded pressures stay
        return sim.boundary_forces()


@pytest.mark.parametrize("nb", [1, 31, 33, 300])
@pytest.mark.parametrize("per_cell", [1, 8, 60])        # rows of 3, 24 and 180 candidates: one load and several
@pytest.mark.parametrize("box", [(0.5, 0.3, 0.3), (3.5, 3.3, 3.4)])      # counting sort's cell ranges and radix sort's
def test_both_forms_give_the_same_forces(nb, per_cell, box):
    n = per_cell * 6 * 6 * 6
    sc = P.dam_break((n, 1, 1), 0.01, box, H, seed=1).replace(n=n, nbr_cap=512)
    rng = np.random.default_rng(nb * 100 + per_cell)
    fluid = rng.uniform(0, 6 * H, (n, 3)).astype(np.float32)
    pressure = rng.uniform(0, 1e4, n).astype(np.float32)
    near = rng.uniform(-0.5 * H, 6.5 * H, (nb, 3)).clip(0).astype(np.float32)      # grid border cells among them
    far = rng.uniform((8 * H, 8 * H, 8 * H), (0.49, 0.29, 0.29), (16384, 3)).astype(np.float32)
    few = forces(sc, fluid, pressure, near)
    many = forces(sc, fluid, pressure, np.concatenate([near, far]))
    assert np.abs(few).max() > 0
    assert np.array_equal(few, many[:nb])
    assert not many[nb:].any()
