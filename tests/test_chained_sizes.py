"""Chained launches (test_chained_launches.py) on both sides of the sizes where
the launches change: from 131,072 particles on the sweeps' blocks over the wall
list are part of a chained launch, from 524,288 threads on launches are not
chained; and of the kinds of step that file leaves out: graphs, the learned
start, batches, training. The same bits as one launch at a time, an event
between any two of them."""
import numpy as np
import pytest

import psb_project_b200 as P

pytestmark = pytest.mark.gpu


def _run(sim, pos, alone, graph, train=False):
    vel = np.random.default_rng(len(pos)).normal(0, 0.1, pos.shape).astype(np.float32)
    sim.set_graph(graph and not alone)                 # steps under the profile are launched one by one
    sim.profile(alone)
    if train:
        sim.mlp_collect(stride=3, capacity=1 << 18)
    for _ in range(2):
        sim.upload(pos, vel, vel)
        sim.step(3)
    out = sim.download()
    if train:
        sim.mlp_collect(0)
        sim.mlp_set_weights(P.mlp_init_weights(0))
        out["loss"] = sim.mlp_train(20, 4096, 2e-3, seed=5)
        out["weights"] = sim.mlp_get_weights()
    return out


def _same(a, b):
    for name in a:
        assert np.array_equal(np.asarray(a[name]), np.asarray(b[name]), equal_nan=True), name


@pytest.mark.parametrize("kind,nxyz,graph", [
    ("plain", (64, 64, 33), False), ("plain", (64, 64, 33), True),         # 135,168: listed
    ("plain", (96, 88, 64), False), ("plain", (96, 88, 64), True),         # 540,672: not chained
    ("learned", (40, 30, 20), False), ("learned", (40, 30, 20), True),
    ("train", (40, 30, 20), False),
])
def test_single_scenes(kind, nxyz, graph):
    box = tuple(round(m * 0.01 * f, 3) for m, f in zip(nxyz, (1.6, 1.4, 1.3)))
    sc = P.dam_break(nxyz, 0.01, box, 0.02, dt=5e-4, seed=2)
    if kind == "learned":
        sc = sc.replace(warm_start=P.WARM_LEARNED)
    out = []
    for alone in (True, False):
        with P.Simulation(sc) as sim:
            if kind == "learned":
                sim.mlp_set_weights(P.mlp_init_weights(4))
            out.append(_run(sim, P.scene_positions(sc), alone, graph, train=kind == "train"))
    _same(*out)


@pytest.mark.parametrize("graph", [False, True])
def test_batches(graph):
    scenes = [P.dam_break((n, 9, 8), 0.01, (n * 0.016 + 0.1, 0.2, 0.2), 0.02, dt=5e-4, seed=n) for n in (3, 17, 90)]
    pos = np.concatenate([P.scene_positions(s) for s in scenes])
    out = []
    for alone in (True, False):
        with P.BatchSimulation(scenes) as sim:
            out.append(_run(sim, pos, alone, graph))
    _same(*out)
