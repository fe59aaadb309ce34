"""GPU parity of fixed-step renders of 20,769 rays around the step length at which they
change from candidate lists to the walk of every step: from a tenth of it to ten times,
and just below and above. Images and search counters equal the oracle's."""
import numpy as np
import pytest

from test_gpu_parity import same_bits
from test_gpu_raylist import TILT, Z, _cluster, _uniform

pytestmark = pytest.mark.gpu

NX, NY = 161, 129
CASES = {
    "seven": (_uniform(7), (50.3, 50.2, 0.0), TILT, 60.0),
    "uniform": (_uniform(3000), (50.3, 50.2, 20.0), Z, 90.0),
    "duplicates": (np.repeat(_uniform(60), 40, axis=0), (50.3, 50.2, 0.0), TILT, 60.0),
    "coded_cells": (_cluster(600, 3.0), (50.0, 50.0, 35.0), TILT, 40.0),
    "outside": (_uniform(3000), (-190.0, 230.0, -350.0), TILT, 300.0),
}


def _line(grid):
    """Step length from which rays are walked (walk_rule in ilc_render.cu)."""
    cell = float(np.mean(grid["cell_sizes"]))
    line = 16384.0 * min(1.0, (grid["num_particles"] / 1048576.0) ** 0.19)
    return 0.28 * cell * line / (NX * NY - line)


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("times,steps", [(0.1, 60), (0.4, 40), (0.98, 25), (1.02, 25), (10.0, 6)])
def test_fixed_steps_around_the_line(ctx, oracle_mod, name, times, steps):
    import illcrawl_b200 as ilc
    pts, pos, look, width = CASES[name]
    ctx.setup_particles(pts)
    depth = times * _line(ctx.grid_describe()) * steps
    g = oracle_mod.Grid(pts)
    args = (pos, look, 0.3, width, NX, NY)
    want, ost = g.render_fixed(oracle_mod.camera(*args), depth, steps)
    img, st = ctx.render_fixed(ilc.camera(*args), depth, steps)
    assert same_bits(img, want)
    assert st["steps"] == NX * NY * steps
    assert st["cells_visited"] == ost[0] and st["candidates"] == ost[1]
