"""Particles near the box faces: their ghost sums against the oracle (every
particle near a face, a few, none at the start but some at the predicted
positions; counts around the warp), with the parity suite's tolerances for
one config-profile step (test_gpu_parity.py); and the wall list that large
contexts use against the plain sweep of small ones, bit for bit."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P
from test_gpu_parity import (TOL, TOL_P_CONFIG_PCI, TOL_V, TOL_V_CONFIG_PCI, _compare_step)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [P.WCSPH, P.PCISPH])
@pytest.mark.parametrize("nxyz,box,shift", [
    ((5, 5, 5), (0.05, 0.05, 0.05), 0.0),       # every face is near
    ((31, 1, 1), (0.4, 0.05, 0.05), 0.0),       # one row along an edge, under a warp
    ((33, 1, 1), (0.4, 0.05, 0.05), 0.0),       # and over one
    ((11, 7, 3), (0.3, 0.3, 0.06), 0.0),        # two faces on z for every particle, corners among them
    ((9, 7, 5), (0.3, 0.3, 0.3), 0.018),        # first layer at 1.15 h: none near a face, some predicted so
])
def test_wall_particles_match_oracle(method, nxyz, box, shift):
    sc = P.dam_break(nxyz, 0.01, box, 0.02, method=method, dt=5e-4, seed=3).replace(warm_start=P.WARM_PREVIOUS)
    rng = np.random.default_rng(4)
    pos = P.scene_positions(sc) + np.float32(shift)
    vel = rng.normal(0, 0.1, pos.shape).astype(np.float32)
    if shift:
        vel -= np.float32(8.0)        # 4 mm in the step's first prediction, 0.2 h
    p = rng.uniform(0, 2000, len(pos)).astype(np.float32) if method == P.PCISPH else None
    sim = P.Simulation(sc)
    sim.upload(pos, vel, vel, p)
    orc = oracle.OracleSim(sc, pos, vel, vel, p, float_state=True)
    sim.step(1)
    so = orc.step()
    if method == P.PCISPH:
        sg = sim.stats()
        if sg.iters != so.iters:      # the deciding error within FP32 rounding of eta
            assert abs(so.err[min(sg.iters, so.iters)] - sc.eta) <= 2e-6
        else:
            _compare_step(sim, orc, pos.astype(np.float64), p_tol=TOL_P_CONFIG_PCI, v_tol=TOL_V_CONFIG_PCI)
    else:
        _compare_step(sim, orc, pos.astype(np.float64), p_tol=TOL, v_tol=TOL_V)
    sim.close()


@pytest.mark.parametrize("nxyz,shift", [((20, 18, 16), 0.0), ((33, 5, 7), 0.0), ((17, 9, 5), 0.018)])
def test_wall_list_matches_plain_sweep(nxyz, shift):
    """A small scene alone (no list) and in a batch of more than 131,072
    particles (listed): the same sums in the same order, so the same bits."""
    small = P.dam_break(nxyz, 0.01, (0.5, 0.4, 0.3), 0.02, dt=5e-4, seed=5).replace(warm_start=P.WARM_PREVIOUS)
    large = P.dam_break((64, 64, 32), 0.01, (1.0, 0.8, 0.4), 0.02, dt=5e-4, seed=6).replace(warm_start=P.WARM_PREVIOUS)
    rng = np.random.default_rng(7)
    state = []
    for sc, d in ((large, 0.0), (small, shift)):
        pos = P.scene_positions(sc) + np.float32(d)
        vel = (rng.normal(0, 0.3, pos.shape) - (6.0 if d else 0.0)).astype(np.float32)
        state.append((pos, vel, vel, rng.uniform(0, 3000, len(pos)).astype(np.float32)))
    with P.BatchSimulation([large, small]) as both, P.Simulation(small) as alone:
        both.upload(*[np.concatenate(a) for a in zip(*state)])
        alone.upload(*state[1])
        both.step(2)
        alone.step(2)
        a, b = both.download(), alone.download()
        first = int(both.first[1])
    for k in b:
        assert np.array_equal(a[k][first:].view(np.uint32), b[k].view(np.uint32)), k
