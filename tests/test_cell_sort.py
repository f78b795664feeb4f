"""The two sorts of a step and the one-block sort, at their edges: integer
work, so every comparison is exact. The grid sort against numpy's stable sort
of the oracle's cell keys, on both sides of the rule that picks counting or
radix (4,194,304 cells), with random, crowded and clamped particles; the
allocation-free entry point around the one-block sort's 8,192 pairs."""
import ctypes

import numpy as np
import pytest

import oracle
import psb_project_b200 as P
from psb_project_b200 import runtime as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 255, 257, 4097, 20000])
@pytest.mark.parametrize("box", [(0.3, 0.2, 0.25), (3.0, 3.5, 3.3)])      # few cells: counting; 4.7M cells: radix
@pytest.mark.parametrize("spread", ["box", "cell", "outside"])
def test_grid_sort_is_stable_by_cell_and_id(n, box, spread):
    sc = P.dam_break((n, 1, 1), 0.01, box, 0.02, seed=1).replace(n=n, nbr_cap=8)
    rng = np.random.default_rng(n)
    lo, hi = {"box": (0.0, 1.0), "cell": (0.5, 0.5), "outside": (-0.5, 1.5)}[spread]
    pos = (rng.uniform(lo, hi, (n, 3)) * np.asarray(box)).astype(np.float32)
    if spread == "cell":
        pos += rng.uniform(0, 0.05, pos.shape).astype(np.float32)        # a few crowded cells
    keys = oracle.cell_keys(sc, pos.astype(np.float64))
    perm = oracle.sort_perm(keys)
    with P.Simulation(sc) as sim:
        for _ in range(2):               # a second build over the first one's words
            sim.upload(pos)
            try:
                sim.build_neighbors()
            except R.PsbError as e:      # crowded cells overflow the short lists; the sort is done
                assert e.status == R.EOVERFLOW_NBR
            assert np.array_equal(sim.read_field(R.FIELD_SORTED_ID), perm)
            assert np.array_equal(sim.read_field(R.FIELD_SORTED_KEY), keys[perm])
            assert np.array_equal(sim.read_field(R.FIELD_CELL_KEY), keys)


@pytest.mark.parametrize("n", [1, 31, 32, 255, 257, 1025, 8191, 8192, 8193])
@pytest.mark.parametrize("bits", [1, 8, 9, 32])
def test_noalloc_sort_sizes(n, bits):
    import torch
    rng = np.random.default_rng(n * 100 + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    vals = rng.permutation(n).astype(np.uint32)
    order = np.argsort(keys, kind="stable")
    dev = lambda a: torch.from_numpy(a.view(np.int32).copy()).cuda()
    k, v = dev(keys), dev(vals)
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    for src, dst in (((k, v), (ko, vo)), ((k, v), (k, v))):              # then in place
        rc = R.lib().psb_sort_cells_noalloc(*[ctypes.c_void_p(t.data_ptr()) for t in src + dst], n, bits,
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == R.OK
        assert np.array_equal(dst[0].cpu().numpy().view(np.uint32), keys[order])
        assert np.array_equal(dst[1].cpu().numpy().view(np.uint32), vals[order])
