"""GPU parity of the per-ray candidate lists (ilc_raylist.cuh) where they can go
wrong: fewer particles than slots, equal distances, one cell holding nearly all
particles (coded scan, lists beyond shared memory), rays outside the grid, views
along cell boundaries, a look-at vector of another length. Image, step counts
and search counters equal the oracle's (bit for bit), through both kernels."""
import numpy as np
import pytest

from test_gpu_parity import same_bits

pytestmark = pytest.mark.gpu

Z = (0.0, 0.0, 1.0)
TILT = (0.48, -0.36, 0.8)


def _uniform(n, seed=3, box=100.0):
    p = np.random.default_rng(seed).random((n, 4)) * box
    p[:, 3] = 1.0 + p[:, 3] / box
    return p.astype(np.float32)


def _cluster(n, sigma, spread=200):
    rng = np.random.default_rng(4)
    p = _uniform(n + spread, seed=5)
    p[:n, :3] = 50.0 + sigma * rng.normal(size=(n, 3))
    return p[rng.permutation(len(p))]


def _lattice(k=9):
    a = np.arange(k) * 11.0 + 3.0
    g = np.stack(np.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
    return np.concatenate([g, 1.0 + g[:, :1] / 100.0], 1).astype(np.float32)


CASES = {
    "one": (_uniform(1), (50.3, 50.2, 0.0), Z, 40.0, 6, 5, 90.0),
    "seven": (_uniform(7), (50.3, 50.2, 0.0), TILT, 60.0, 6, 5, 90.0),
    "eight": (_uniform(8), (50.3, 50.2, 0.0), Z, 60.0, 6, 5, 90.0),
    "hundred": (_uniform(100), (20.3, 60.2, 5.0), TILT, 60.0, 9, 7, 120.0),
    "duplicates": (np.repeat(_uniform(60), 40, axis=0), (50.3, 50.2, 0.0), TILT, 60.0, 8, 8, 90.0),
    # rays through particles: equal distances, and a point exactly on a particle
    "lattice_on": (_lattice(), (47.0, 47.0, 2.0), Z, 88.0, 8, 8, 60.0),
    "lattice_offset": (_lattice(), (50.17, 50.09, 1.0), Z, 52.0, 8, 8, 60.0),
    "dense_384": (_cluster(384, 0.4), (50.0, 50.0, 44.0), Z, 4.0, 8, 8, 12.0),
    "dense_3000": (_cluster(3000, 0.3), (50.0, 50.0, 47.0), TILT, 2.0, 8, 8, 6.0),
    "dense_20000": (_cluster(20000, 0.3), (50.0, 50.0, 48.5), Z, 2.0, 8, 4, 3.0),
    "outside": (_uniform(3000), (-190.0, 230.0, -350.0), TILT, 300.0, 9, 9, 1000.0),
    "far_origin": (_uniform(3000) + np.float32([30000, -20000, 9000, 0]),
                   (30050.0, -19950.0, 9000.0), TILT, 80.0, 9, 9, 150.0),
    "long_look": (_uniform(3000), (50.3, 50.2, 0.0), tuple(2.0 * v for v in TILT), 60.0, 8, 8,
                  60.0),
    "diagonal": (_uniform(3000), (0.0, 0.0, 0.0), (3 ** -0.5,) * 3, 20.0, 8, 8, 170.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_ray_lists_bit_exact(ctx, oracle_mod, name):
    import illcrawl_b200 as ilc
    pts, pos, look, width, nx, ny, depth = CASES[name]
    ctx.setup_particles(pts)
    g = oracle_mod.Grid(pts)
    args = (pos, look, 0.0 if name == "lattice_on" else 0.3, width, nx, ny)
    out, steps, acc, ost, rc = g.render(oracle_mod.camera(*args), depth, 0.0, 1e-3, mode=1)
    assert rc == 0
    img, st = ctx.render_adaptive(ilc.camera(*args), depth, 1e-3, 0.0, 1)
    gimg, rs, gst = ctx.render_ray_stats(ilc.camera(*args), depth, 1e-3, 0.0, 1)
    for a, s in ((img, st), (gimg, gst)):
        assert same_bits(a, out)
        assert s["steps"] == steps.sum() and s["accepted_steps"] == acc.sum()
        assert s["cells_visited"] == ost[0] and s["candidates"] == ost[1]
    assert np.array_equal(rs[:, 0], steps) and np.array_equal(rs[:, 1], acc)
    # steps long against the cells and short against them
    for n in (3, 200):
        fo, _ = g.render_fixed(oracle_mod.camera(*args), depth, n)
        assert same_bits(ctx.render_fixed(ilc.camera(*args), depth, n)[0], fo)
    # a value table in place of the particles' own values
    vals = (pts[:, 3] * 0.5 + pts[:, 0] * 1e-3).astype(np.float32)
    jobs = [ilc.job(ilc.camera(*args), z_range=depth)]
    ojobs = [oracle_mod.job(oracle_mod.camera(*args), z_range=depth)]
    for v in (vals, np.stack([vals, 2.0 * vals, vals * vals], 1)):
        bout, _ = ctx.render_batched(v, jobs)
        want, _, rc = oracle_mod.render_batched(g, v, ojobs, 0.0, 1e-3)
        assert rc == 0 and same_bits(bout, want)
