"""GPU parity of fixed-step renders on both sides of the line between the two
fixed-step kernels (image sides that are no multiples of the 16 x 8 tiles): few
long steps over 20,769 rays walk every step from scratch, 24 short ones go
through candidate lists. Images and search counters equal the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import same_bits
from test_gpu_raylist import TILT, Z, _cluster, _uniform

pytestmark = pytest.mark.gpu

CASES = {
    "seven": (_uniform(7), (50.3, 50.2, 0.0), TILT, 60.0, 300.0),
    "uniform": (_uniform(3000), (50.3, 50.2, 0.0), Z, 90.0, 90.0),
    "uniform_tilt": (_uniform(3000), (20.3, 60.2, 5.0), TILT, 60.0, 120.0),
    "duplicates": (np.repeat(_uniform(60), 40, axis=0), (50.3, 50.2, 0.0), TILT, 60.0, 120.0),
    "coded_cells": (_cluster(600, 3.0), (50.0, 50.0, 0.0), TILT, 40.0, 120.0),
    "outside": (_uniform(3000), (-190.0, 230.0, -350.0), TILT, 300.0, 1000.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("steps", [1, 3, 24])
def test_fixed_steps_bit_exact(ctx, oracle_mod, name, steps):
    import illcrawl_b200 as ilc
    pts, pos, look, width, depth = CASES[name]
    ctx.setup_particles(pts)
    g = oracle_mod.Grid(pts)
    args = (pos, look, 0.3, width, 161, 129)
    want, ost = g.render_fixed(oracle_mod.camera(*args), depth, steps)
    img, st = ctx.render_fixed(ilc.camera(*args), depth, steps)
    assert same_bits(img, want)
    assert st["steps"] == 161 * 129 * steps
    assert st["cells_visited"] == ost[0] and st["candidates"] == ost[1]
