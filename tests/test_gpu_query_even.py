"""GPU parity of nn8 queries where nearly all grid cells hold particles and hardly
any of them many, on both sides of the rule that takes them there (one warp per
query below 24,576, one lane per query in the given order from there on, in the
order of their bins from 393,216 on): slots, distances, values and search counters
equal the oracle's, also with distances that tie, with a cell that is left to the
warps, with queries on particles and outside the grid, and when a second block is
merged. The number of kernel launches shows the way taken."""
import numpy as np
import pytest

from test_gpu_parity import same_bits
from test_gpu_query_paths import _queries
from test_gpu_raylist import _uniform

pytestmark = pytest.mark.gpu


def _crowd(k):
    """Uniform particles and a cell of some k more."""
    p = _uniform(100_000)
    p[:k, :3] = 50.0 + 0.2 * np.random.default_rng(8).normal(size=(k, 3)).astype(np.float32)
    return p


SETS = {"uniform": lambda: _uniform(30_000), "thousand": lambda: _uniform(1000),
        "duplicates": lambda: np.repeat(_uniform(10_000), 3, axis=0), "crowd": lambda: _crowd(120),
        "more_crowd": lambda: _crowd(200)}
# one launch: warps; two: lanes, then warps for the rest; more: count, scan and order first
LAUNCHES = {24_575: 1, 24_576: 2, 393_215: 2}


@pytest.mark.parametrize("n", [24_575, 24_576, 393_215, 393_216])
@pytest.mark.parametrize("name", sorted(SETS))
def test_query_even_bit_exact(ctx, oracle_mod, name, n):
    pts = SETS[name]()
    q = _queries(n, pts)
    ctx.setup_particles(pts)
    cells = ctx.grid_export()[0]
    held = cells[:, 1] - cells[:, 0]
    crowd = int(np.maximum(held - 48, 0).sum())
    assert np.count_nonzero(held) >= 0.8 * len(held)
    assert (crowd > len(pts) // 1024) == (name == "more_crowd") and (crowd > 0) == ("crowd" in name)
    before = ctx.kernel_launches
    val, idx, d8 = ctx.nn8_query(q, slots=True)
    launches = ctx.kernel_launches - before
    stats = ctx.last_query_stats()
    if name == "more_crowd":
        assert launches == 1 if n < 81_920 else launches > 4
    else:
        assert launches == LAUNCHES.get(n, launches) and (n in LAUNCHES or launches > 4)
    oval, oidx, od8, ost = oracle_mod.Grid(pts).nn8(q)
    assert np.array_equal(idx, oidx)
    assert same_bits(d8, od8)
    assert same_bits(val, oval)
    assert stats == (int(ost[0]), int(ost[1]))


@pytest.mark.parametrize("n", [24_576, 393_216])
def test_query_even_merge(ctx, oracle_mod, n):
    pts = np.random.default_rng(9).permutation(_crowd(200))
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
