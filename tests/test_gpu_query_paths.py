"""GPU parity of nn8 queries on both sides of the rule that picks their kernel
(one warp per query below 81,920 queries, one lane per query from there on with
the dense ones left to the warp kernel): slots, distances, values and search
counters equal the oracle's, also where distances tie, where one cell holds
nearly all particles, outside the grid, and when a second block is merged."""
import numpy as np
import pytest

from conftest import random_queries
from test_gpu_parity import same_bits
from test_gpu_raylist import _cluster, _lattice, _uniform

pytestmark = pytest.mark.gpu

SETS = {
    "seven": lambda: _uniform(7),
    "uniform": lambda: _uniform(30_000),
    "duplicates": lambda: np.repeat(_uniform(600), 30, axis=0),
    "lattice": lambda: _lattice(),
    "cells_of_97": lambda: np.repeat(_uniform(97), 160, axis=0),
    "dense_cell": lambda: _cluster(4000, 0.5),
}


def _queries(n, pts):
    q = random_queries(n, -20.0, 120.0, seed=n)
    k = min(n // 2, len(pts))
    q[:k, :3] = pts[:k, :3]                       # on particles
    q[k:k + k // 2, :3] = pts[:k // 2, :3] + np.float32(0.25)
    if n > 20:
        q[-1, :3] = np.nan
        q[-2, :3] = [1e30, -1e30, 0.0]
    return q


@pytest.mark.parametrize("n", [1, 33, 81_919, 81_920])
@pytest.mark.parametrize("name", sorted(SETS))
def test_query_paths_bit_exact(ctx, oracle_mod, name, n):
    pts = SETS[name]()
    q = _queries(n, pts)
    ctx.setup_particles(pts)
    val, idx, d8 = ctx.nn8_query(q, slots=True)
    cells, cands = ctx.last_query_stats()
    oval, oidx, od8, ost = oracle_mod.Grid(pts).nn8(q)
    assert np.array_equal(idx, oidx)
    assert same_bits(d8, od8)
    assert same_bits(val, oval)
    assert (cells, cands) == (int(ost[0]), int(ost[1]))


@pytest.mark.parametrize("n", [500, 81_920])
def test_query_paths_merge(ctx, oracle_mod, n):
    pts = _cluster(4000, 0.5, spread=6000)
    a, b = pts[: len(pts) // 2], pts[len(pts) // 2:]
    q = _queries(n, pts)
    ctx.setup_particles(a)
    first = ctx.nn8_query(q)
    ctx.setup_particles(b)
    merged = ctx.nn8_query(q, merge_previous=True)
    o1, lists = oracle_mod.nn8_lists(oracle_mod.Grid(a), q)
    o2, lists = oracle_mod.nn8_lists(oracle_mod.Grid(b), q, merge=True, lists=lists)
    assert same_bits(first, o1)
    assert same_bits(merged, o2)
