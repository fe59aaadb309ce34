"""GPU parity of adaptive renders of many rays, which are walked step by step while
their steps are long against a cell and left to the candidate lists otherwise: tight
and loose tolerances (all rays left, some, none), a dense cell on the way, rays
outside the grid, apertures and chords, both controllers, value tables and several
channels, recorded and replayed steps, the step limit. Images, step counts and search
counters equal the oracle's; the number of kernel launches (walk, list of the rays
left, lists) shows that rays were walked."""
import numpy as np
import pytest

from test_gpu_parity import same_bits
from test_gpu_raylist import TILT, Z, _cluster, _uniform

pytestmark = pytest.mark.gpu

NX, NY = 197, 129  # no multiples of the 16 x 8 tiles
CASES = {
    "seven": (_uniform(7), (50.3, 50.2, 0.0), TILT, 60.0, 300.0),
    "uniform": (_uniform(3000), (50.3, 50.2, 0.0), Z, 90.0, 90.0),
    "uniform_tilt": (_uniform(3000), (20.3, 60.2, 5.0), TILT, 60.0, 120.0),
    "duplicates": (np.repeat(_uniform(60), 40, axis=0), (50.3, 50.2, 0.0), TILT, 60.0, 120.0),
    "coded_cells": (_cluster(600, 3.0), (50.0, 50.0, 0.0), TILT, 40.0, 120.0),
    "dense": (_cluster(6000, 0.8), (50.0, 50.0, 0.0), Z, 60.0, 100.0),
    "outside": (_uniform(3000), (-190.0, 230.0, -350.0), TILT, 300.0, 1000.0),
}


def _setup(ctx, oracle_mod, name):
    pts, pos, look, width, depth = CASES[name]
    ctx.setup_particles(pts)
    return pts, oracle_mod.Grid(pts), (pos, look, 0.3, width, NX, NY), depth


@pytest.mark.parametrize("rtol", [1e-1, 1e-2, 2e-3])
@pytest.mark.parametrize("name", sorted(CASES))
def test_adaptive_walk_bit_exact(ctx, oracle_mod, name, rtol):
    import illcrawl_b200 as ilc
    pts, g, args, depth = _setup(ctx, oracle_mod, name)
    cam, ocam = ilc.camera(*args), oracle_mod.camera(*args)
    for controller in (0, 1):
        out, steps, acc, ost, rc = g.render(ocam, depth, 0.0, rtol, mode=controller)
        assert rc == 0
        before = ctx.kernel_launches
        img, st = ctx.render_adaptive(cam, depth, rtol, 0.0, controller)
        # (the job table's cost order is a launch of its own)
        assert ctx.kernel_launches - before == 3 + (controller == 1)
        gimg, rs, gst = ctx.render_ray_stats(cam, depth, rtol, 0.0, controller)
        for a, s in ((img, st), (gimg, gst)):
            assert same_bits(a, out)
            assert s["steps"] == steps.sum() and s["accepted_steps"] == acc.sum()
            assert s["cells_visited"] == ost[0] and s["candidates"] == ost[1]
        assert np.array_equal(rs[:, 0], steps) and np.array_equal(rs[:, 1], acc)


@pytest.mark.parametrize("name", ["uniform_tilt", "coded_cells", "dense"])
def test_adaptive_walk_record_and_replay(ctx, oracle_mod, name):
    import illcrawl_b200 as ilc
    pts, g, args, depth = _setup(ctx, oracle_mod, name)
    cam, ocam = ilc.camera(*args), oracle_mod.camera(*args)
    out, ohs, on, rc = g.render_record(ocam, depth, 0.0, 1e-2, mode=1, cap=600)
    assert rc == 0
    img, hs, n, st = ctx.render_record(cam, depth, 600, 1e-2)
    assert same_bits(img, out) and np.array_equal(n, on)
    k = np.arange(600)[None, :] < on[:, None]
    assert same_bits(hs[k], ohs[k])
    before = ctx.kernel_launches
    frozen, fst = ctx.render_frozen(cam, depth, ohs, on)
    assert ctx.kernel_launches - before == 3
    assert same_bits(frozen.ravel(), g.render_replay(ocam, ohs, on))
    assert fst["steps"] == on.sum()


@pytest.mark.parametrize("tile_w", [8, 0])
@pytest.mark.parametrize("rtol", [3e-2, 3e-3])
def test_adaptive_walk_jobs(ctx, oracle_mod, rtol, tile_w):
    """Cameras with apertures and chords; one channel and several (lanes with one
    group of four, with none, with several)."""
    import illcrawl_b200 as ilc
    pts, g, args, depth = _setup(ctx, oracle_mod, "coded_cells")
    rng = np.random.default_rng(3)

    def jobs(m):
        cam = m.camera
        return [m.job(cam(*args), z_range=depth),
                m.job(cam((50.0, 50.0, -10.0), Z, 0.1, 90.0, 70, 50), aperture_radius=30.0,
                      sphere_center=(50.0, 50.0, 50.0), sphere_radius=40.0, min_chord=5.0)]

    ctx.set_batch_schedule(tile_w=tile_w)
    try:
        for v in (1, 3, 4, 136):
            vals = (0.5 + rng.random((len(pts), v))).astype(np.float32)
            vals = vals[:, 0] if v == 1 else vals
            before = ctx.kernel_launches
            img, st = ctx.render_batched(vals, jobs(ilc), rel_tol=rtol)
            # channel sort, cost of two jobs, walk, left rays, lists
            assert ctx.kernel_launches - before == 6
            ojobs = jobs(oracle_mod)
            ojobs[1].out_offset = v * NX * NY
            want, ost, rc = oracle_mod.render_batched(g, vals, ojobs, 0.0, rtol)
            assert rc == 0 and same_bits(img, want)
    finally:
        ctx.set_batch_schedule()


def test_chords_take_lists(ctx, oracle_mod):
    """Rays on chords through a core are not walked first, however many they are."""
    import illcrawl_b200 as ilc
    pts, g, args, depth = _setup(ctx, oracle_mod, "coded_cells")
    vals = pts[:, 3].copy()

    def jobs(m):
        return [m.job(m.camera((50.0, 50.0, -10.0), Z, 0.1, 90.0, NX, NY), aperture_radius=44.0,
                      sphere_center=(50.0, 50.0, 50.0), sphere_radius=40.0, min_chord=5.0)]

    before = ctx.kernel_launches
    img, st = ctx.render_batched(vals, jobs(ilc), rel_tol=2e-2)
    assert ctx.kernel_launches - before == 3  # channel sort, cost, lists
    want, ost, rc = oracle_mod.render_batched(g, vals, jobs(oracle_mod), 0.0, 2e-2)
    assert rc == 0 and same_bits(img, want)


def test_adaptive_walk_step_limit(ctx, oracle_mod):
    """Rays that reach the step limit are reported, walked or not."""
    import illcrawl_b200 as ilc
    pts, g, args, depth = _setup(ctx, oracle_mod, "uniform_tilt")
    try:
        for limit in (1, 5, 12):
            ctx.set_step_limit(limit)
            for controller in (0, 1):
                with pytest.raises(ilc.IlcError) as e:
                    ctx.render_adaptive(ilc.camera(*args), depth, 1e-3, 0.0, controller)
                assert e.value.status == 6
    finally:
        ctx.set_step_limit(1 << 20)


@pytest.mark.parametrize("controller", [0, 1])
def test_adaptive_walk_adjoint(ctx, gaunt_table, controller):
    """Image and gradient of many rays, walked in both passes, against those of bands
    of 8 rows, which go through the lists: the same terms, added in another order."""
    import illcrawl_b200 as ilc
    from illcrawl_b200 import synthetic
    c = synthetic.small_cells(4000, seed=43, box=400.0, r_s=50.0)
    ctx.load_gaunt()
    cells = c.xyzq(np.zeros(c.n, np.float32))
    cam = ilc.camera((200, 200, 0), TILT, 0.2, 300.0, NX, NY)
    rng = np.random.default_rng(5)
    target = np.exp(rng.normal(size=(NY, NX)) - 20.0).astype(np.float32)
    args = (cells, c.rho, c.u, c.xe, cam, 400.0, target)
    out = {}
    try:
        for name, mode, budget in (("bands", 0, 1), ("checkpoint", 0, 0), ("recompute", 1, 0)):
            ctx.set_checkpoint_budget(budget)
            before = ctx.kernel_launches
            out[name] = ctx.adjoint_xray_flux(*args, mode=mode, rel_tol=1e-2,
                                              controller=controller)
            out[name] += (ctx.kernel_launches - before,)
    finally:
        ctx.set_checkpoint_budget(0)
    img, g_rho, g_t, st, _ = out["bands"]
    for name in ("checkpoint", "recompute"):
        i, r, t, s, launches = out[name]
        # one band: walk, list of the rays left, lists, then walk and lists
        assert launches == out["recompute"][4]
        assert same_bits(i, img)
        assert s["forward_steps"] == st["forward_steps"]
        assert s["loss"] == pytest.approx(st["loss"], rel=1e-12)
        # sums of up to 1e7 terms in double (1e-9 of their size), rounded to float
        for a, b in ((r, g_rho), (t, g_t)):
            size = np.abs(b).max()
            assert size > 0 and np.isfinite(b).all()
            assert np.all(np.abs(a - b) <= 2e-7 * np.abs(b) + 1e-9 * size)
    # every band has a launch for the render and the adjoint at least
    assert out["bands"][4] > out["checkpoint"][4]
