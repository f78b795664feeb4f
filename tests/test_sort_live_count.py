"""A context whose grid is large for the particles it holds sorts by radix and
one that holds many by counting, whatever its capacity: the sort follows the
live count through uploads and emissions, each change over the other form's
cell words. Sorted order exact against numpy's stable sort of the oracle's
keys; neighbour counts and densities those of a context with a small grid."""
import numpy as np
import pytest

import oracle
import psb_project_b200 as P
from psb_project_b200 import runtime as R

pytestmark = pytest.mark.gpu

CELLS = (465, 465, 466)              # 100.8M: counting from ~61,000 particles on
CAPACITY = 4_200_000


def _check(sim, pos, counting):
    sim.profile_reset()
    sim.build_neighbors()
    ran = {name for name, (launches, _) in sim.profile_read().items() if launches}
    assert ("radix_sort" in ran) == (not counting) and ("cell_sort" in ran or "cell_place" in ran) == counting
    keys = oracle.cell_keys(sim.scene, pos.astype(np.float64))
    assert np.array_equal(sim.read_field(R.FIELD_SORTED_ID), oracle.sort_perm(keys))
    assert np.array_equal(sim.read_field(R.FIELD_CELL_KEY), keys)
    small = sim.scene.replace(n=len(pos), dims=tuple(int(np.ceil((m + 0.02) / sim.scene.cell)) + 2 for m in pos.max(0)))
    with P.Simulation(small) as s:
        s.upload(pos)
        s.build_neighbors()
        for f in (R.FIELD_NBR_COUNT, R.FIELD_DENSITY_X):
            assert np.array_equal(sim.read_field(f), s.read_field(f))


@pytest.mark.parametrize("method", [P.WCSPH, P.PCISPH])
def test_sort_follows_the_live_count(method):
    box = tuple(0.02 * (d - 2) for d in CELLS)
    sc = P.dam_break((80, 60, 63), 0.01, box, 0.02, method=method, dt=1e-4, seed=3, jitter=1e-3, nbr_cap=64)
    pos = P.scene_positions(sc)
    n = len(pos)                     # 302,400
    few, most = 5000, 40_000
    with P.Simulation(sc.replace(n=CAPACITY, dims=CELLS)) as sim:
        sim.profile(True)
        for k in (few, n, few):      # an upload on each side of the line, and back
            sim.upload(pos[:k])
            _check(sim, pos[:k], counting=k == n)
        sim.upload(pos[:most])
        _check(sim, pos[:most], counting=False)
        sim.emit(pos[most:])         # over the line in mid-run
        _check(sim, pos, counting=True)
