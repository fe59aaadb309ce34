"""GPU parity of renders whose camera is thousands of box lengths away, where a
position along a ray is known to a fraction of a cell only: the candidate lists of
a ray segment must end before the rounding of the ray takes a point into the next
subcell. Images and search counters equal the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import same_bits
from test_gpu_raylist import _uniform

pytestmark = pytest.mark.gpu

LOOKS = {"tilt": (0.48, -0.36, 0.8), "y": (0.0, 0.8, 0.6)}


@pytest.mark.parametrize("look", sorted(LOOKS))
@pytest.mark.parametrize("lengths", [50, 1000, 3000, 5000, 20000])
def test_far_camera_bit_exact(ctx, oracle_mod, look, lengths):
    import illcrawl_b200 as ilc
    pts = _uniform(3000)
    v, dist = LOOKS[look], 100.0 * lengths
    pos = tuple(50.0 - dist * k for k in v)
    nx, ny, m = 33, 27, 50
    args = (pos, v, 0.3, 90.0, nx, ny)
    # one step to somewhere in the box, then short ones (frozen: an adaptive ray
    # cannot end where a step's last 0.01 is below the rounding of z)
    hs = np.full((nx * ny, m), 0.37, np.float32)
    hs[:, 0] = dist - 55.0 + 80.0 * np.random.default_rng(7).random(nx * ny)
    n = np.full(nx * ny, m, np.int32)
    ctx.setup_particles(pts)
    g = oracle_mod.Grid(pts)
    cam = ilc.camera(*args)
    want = g.render_replay(oracle_mod.camera(*args), hs, n)
    img, st = ctx.render_frozen(cam, dist + 100.0, hs, n)
    assert st["steps"] == nx * ny * m
    # the search counters of every step's four points, located on their own
    plane = ilc.camera_plane(cam)
    f = np.float32
    tx, ty = (np.arange(k, dtype=f) * plane[12] for k in (nx, ny))
    z = np.zeros(nx * ny, f)
    pts4 = []
    for k in range(m):
        h = hs[:, k]
        for c in (f(3) / f(8), f(12) / f(13), f(1), f(0.5)):
            zq = z + c * h
            q = np.zeros((ny, nx, 4), f)
            for a in range(3):
                o = (plane[9 + a] + tx[None, :] * plane[3 + a]) + ty[:, None] * plane[6 + a]
                q[..., a] = o + zq.reshape(ny, nx) * plane[a]
            pts4.append(q.reshape(-1, 4))
        z = z + h
    cells, cands = g.nn8(np.concatenate(pts4), slots=False)[-1][:2]
    assert (st["cells_visited"], st["candidates"]) == (int(cells), int(cands))
    assert same_bits(img.ravel(), want)
