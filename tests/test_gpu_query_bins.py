"""GPU parity of nn8 queries that are taken in the order of their bins where the
bins are hard to number: grids whose cells and subcells outnumber the bins (several
cells to a bin), queries at, past and far past every face, and an axis of more than
2^23 cells, on which the last half cell's index has no float of its own. Slots,
distances, values and search counters equal the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import same_bits

pytestmark = pytest.mark.gpu

N_QUERIES = 81_920  # the fewest that are ordered


def _line():
    """29,786 particles on a line: 8,414,224 x 1 x 1 cells of 9.5."""
    rng = np.random.default_rng(11)
    p = np.zeros((29_786, 4), np.float32)
    p[:, 0] = np.sort(rng.random(len(p))) * 8e7
    p[0, 0], p[-1, 0] = 0.0, 8e7
    p[:, 3] = 1.0 + rng.random(len(p))
    return p, (0.0, 8e7), 5.0


def _plate():
    """Particles of a thin plate: 2.4 million cells."""
    rng = np.random.default_rng(12)
    p = (rng.random((200_000, 4)) * [3e4, 3e4, 1e-3, 1.0] + [0, 0, 0, 1.0]).astype(np.float32)
    return p, (0.0, 3e4), 40.0


@pytest.mark.parametrize("make", [_line, _plate])
def test_query_bins_bit_exact(ctx, oracle_mod, make):
    pts, (lo, hi), thick = make()
    rng = np.random.default_rng(13)
    q = np.zeros((N_QUERIES, 4), np.float32)
    q[:, 0] = lo + rng.random(len(q)) * (hi - lo)
    q[:, 1] = (lo + rng.random(len(q)) * (hi - lo)) if make is _plate else \
        rng.uniform(-thick, thick, len(q))
    q[:, 2] = rng.uniform(-thick, thick, len(q))
    q[:2000, 0] = hi + rng.uniform(-20.0, 100.0, 2000)     # the upper end of the long axis
    q[2000:3000, 0] = lo - rng.uniform(0.0, 100.0, 1000)
    q[3000:4000, 0] = pts[rng.integers(0, len(pts), 1000), 0]
    q[4000, 0], q[4001, 0], q[4002, 0] = 1e30, -1e30, np.nan
    ctx.setup_particles(pts)
    total = ctx.grid_describe()["total_cells"]
    assert 8 * total > 1 << 20
    if make is _line:
        assert total == 8_414_224
    val, idx, d8 = ctx.nn8_query(q, slots=True)
    cells, cands = ctx.last_query_stats()
    oval, oidx, od8, ost = oracle_mod.Grid(pts).nn8(q)
    assert np.array_equal(idx, oidx)
    assert same_bits(d8, od8)
    assert same_bits(val, oval)
    assert (cells, cands) == (int(ost[0]), int(ost[1]))
