"""Kernels placed behind one another's tails compute what they compute one at
a time. With the profile on, an event stands between any two launches, so no
launch overlaps another: the state after some steps has to be the same to the
bit, for every step kind, on both sides of the warp, block and chip sizes."""
import numpy as np
import pytest

import psb_project_b200 as P

pytestmark = pytest.mark.gpu

KINDS = {
    "wcsph": lambda n: P.dam_break((n, 8, 9), 0.02, (n * 0.02 + 0.3, 0.4, 0.4), 0.04, method=P.WCSPH, dt=2e-4),
    "pcisph": lambda n: P.dam_break((n, 8, 9), 0.02, (n * 0.02 + 0.3, 0.4, 0.4), 0.04, dt=5e-4),
    "reference": lambda n: P.dam_break((n, 8, 9), 0.02, (n * 0.02 + 0.3, 0.4, 0.4), 0.04, dt=5e-4,
                                       profile=P.PROFILE_REF),
    "dem": lambda n: P.dem_block((n, 8, 9), 0.0195, (0.0, 0.0, 0.0), (n * 0.02 + 0.3, 0.4, 0.4), 0.01, dt=1e-4),
}


@pytest.mark.parametrize("n", [1, 5, 60, 900])            # 72 particles to 64,800
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("graph", [False, True])
def test_same_state_as_one_launch_at_a_time(kind, n, graph):
    sc = KINDS[kind](n)
    out = []
    for alone in (True, False):
        with P.Simulation(sc) as sim:
            pos = P.scene_positions(sc)
            vel = np.random.default_rng(n).normal(0, 0.1, pos.shape).astype(np.float32)
            if graph and not alone and kind == "pcisph":
                sim.set_graph(True)
            sim.profile(alone)
            for _ in range(2):                            # a second upload over the first one's words
                sim.upload(pos, vel, vel)
                sim.step(6)
            out.append(sim.download())
    for name in out[0]:
        assert np.array_equal(np.asarray(out[0][name]), np.asarray(out[1][name]), equal_nan=True), name
