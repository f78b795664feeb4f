"""The wall list of single scenes (from 131,072 particles on) against the plain
sweep: one more particle, alone in its neighbourhood, crosses the line, and
leaves every other particle's sums and their order the same, so the same bits;
with it the reorder changes from one launch to two. Every kind of sweep with
ghost terms: WCSPH, PCISPH from zero, from the carried pressure beside a
static and a moving solid, and with the network's inputs."""
import numpy as np
import pytest

import psb_project_b200 as P

pytestmark = pytest.mark.gpu

NXYZ, BOX = (64, 64, 32), (0.9, 0.8, 0.36)


@pytest.mark.parametrize("kind", ["wcsph", "zero", "solid", "moving", "learned"])
def test_list_and_plain_sweep_give_the_same_bits(kind):
    warm = {"solid": P.WARM_PREVIOUS, "moving": P.WARM_PREVIOUS, "learned": P.WARM_LEARNED}.get(kind, P.WARM_ZERO)
    sc = P.dam_break(NXYZ, 0.01, BOX, 0.02, method=P.WCSPH if kind == "wcsph" else P.PCISPH, seed=3, jitter=1e-3,
                     dt=2e-4 if kind == "wcsph" else 5e-4).replace(warm_start=warm)
    pos = P.scene_positions(sc)
    n = len(pos) - 1                                   # 131,071: one short of the list
    pos[n] = (0.85, 0.75, 0.33)                        # over the floor beside the block, 0.2 m from it
    rng = np.random.default_rng(8)
    vel = rng.normal(0, 0.2, pos.shape).astype(np.float32)
    vel[n] = 0
    p = rng.uniform(0, 2000, len(pos)).astype(np.float32)
    solid = P.sphere_shell((0.72, 0.06, 0.18), 0.06, 0.01)
    out = []
    for m in (n, n + 1):
        with P.Simulation(sc) as sim:
            if kind in ("solid", "moving"):
                sim.set_boundary(solid)
            if kind == "learned":
                sim.mlp_set_weights(P.mlp_init_weights(4))
            sim.upload(pos[:m], vel[:m], vel[:m], None if kind == "wcsph" else p[:m])
            if kind == "moving":
                sim.set_boundary_motion(np.zeros_like(solid), np.zeros_like(solid), 2e-3)
            sim.step(3)
            out.append((sim.download(), sim.stats().iters_total))
    assert out[0][1] == out[1][1]
    for name, a in out[0][0].items():
        assert np.array_equal(a.view(np.uint32), out[1][0][name][:n].view(np.uint32)), name
