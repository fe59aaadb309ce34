"""The autotuners launch each distinct schedule once: the z window has no effect, and
occupancies above what is resident are the same launch. Times of one launch stand for
all candidates that come to it, and the first of those is returned."""
import numpy as np
import pytest

from test_gpu_raylist import Z, _uniform

pytestmark = pytest.mark.gpu

ARGS = ((50.3, 50.2, 0.0), Z, 0.0, 90.0, 48, 40)


def test_autotune_render_times_distinct_launches(ctx):
    import illcrawl_b200 as ilc
    ctx.setup_particles(_uniform(3000))
    before = ctx.kernel_launches
    try:
        bw, bo, times = ctx.autotune_render(ilc.camera(*ARGS), 90.0, 1e-2, windows=(20, 0, 5),
                                            occupancies=(5, 0, 4, 3), sample_stride=1)
        assert ctx.kernel_launches - before == 2  # as many blocks as fit (4), and 3
        assert bw == 20.0 and bo in (5, 3)
        for o in (5, 0, 4, 3):
            assert len({times[(w, o)] for w in (20.0, 0.0, 5.0)}) == 1
        assert times[(0.0, 5)] == times[(0.0, 0)] == times[(0.0, 4)]
        assert times[(bw, bo)] == min(times.values()) > 0
        with pytest.raises(ilc.IlcError):
            ctx.autotune_render(ilc.camera(*ARGS), 90.0, 1e-2, windows=(0, -1))
        with pytest.raises(ilc.IlcError):
            ctx.autotune_render(ilc.camera(*ARGS), 90.0, 1e-2, occupancies=(4, 2))
    finally:
        ctx.set_render_occupancy(4)


@pytest.mark.parametrize("channels", [1, 5])
def test_autotune_batched_times_distinct_launches(ctx, channels):
    import illcrawl_b200 as ilc
    pts = _uniform(3000)
    ctx.setup_particles(pts)
    vals = np.repeat(pts[:, 3:], channels, axis=1)
    vals = vals[:, 0] if channels == 1 else vals
    jobs = [ilc.job(ilc.camera(*ARGS), z_range=90.0)]
    before = ctx.kernel_launches
    try:
        bt, bo, bw, times = ctx.autotune_batched(vals, jobs, rel_tol=1e-2, tile_ws=(4, 0),
                                                 occupancies=(0, 3, 4), windows=(7.0, 0.0))
        # at most 4 blocks of any kernel fit; channel sort, cost and render each
        assert ctx.kernel_launches - before == 2 * 2 * 3
        assert bw == 7.0 and bt in (4, 0) and bo in (0, 3)
        for t in (4, 0):
            for o in (0, 3, 4):
                assert times[(t, o, 7.0)] == times[(t, o, 0.0)] > 0
            assert times[(t, 0, 0.0)] == times[(t, 4, 0.0)]
        assert times[(bt, bo, bw)] == min(times.values())
    finally:
        ctx.set_batch_schedule()
