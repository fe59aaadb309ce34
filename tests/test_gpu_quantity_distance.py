"""GPU parity of the per-cell quantities over luminosity distances: those of redshifts
from 0 to 10 in kpc and Mpc, and both sides of the limits between which the emission's
division by the distance squared goes through its reciprocal. Bit for bit against the
oracle."""
import numpy as np
import pytest

from test_gpu_parity import same_bits
from test_gpu_quantity_edges import DX, X0, Z, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist", [0.9e-10, 1.1e-10, 1e-9, 2e-7, 4.3, 1.06e5, 3.1e7, 3.3e7, 1.06e8,
                                  0.99e10, 1.01e10])
def test_quantities_distances(ctx, oracle_mod, gaunt_table, dist):
    from illcrawl_b200 import synthetic
    ctx.load_gaunt()
    arf = synthetic.synthetic_arf(n=130)
    ctx.load_arf(arf, X0, DX)
    rho, u, xe = _inputs(3000, 71)
    assert same_bits(ctx.xray_flux(rho, u, xe, Z, dist, 0.5, 7.0, 100),
                     oracle_mod.xray_band(gaunt_table, rho, u, xe, Z, dist, 0.5, 7.0, 100))
    assert same_bits(ctx.xray_photon_flux(rho, u, xe, Z, dist, 0.1, 10.0, 100),
                     oracle_mod.xray_photon_flux(gaunt_table, rho, u, xe, Z, dist, 0.1, 10.0, 100))
    assert same_bits(ctx.chandra_count_rate(rho, u, xe, Z, dist),
                     oracle_mod.chandra_count_rate(gaunt_table, arf, X0, DX, rho, u, xe, Z, dist))
    e, w = np.float32([0.3, 1.0, 9.0]), np.float32([0.1, 0.2, 0.5])
    x = ctx.xray_spectrum(rho, u, xe, e, w, Z, dist)
    for b in range(3):
        assert same_bits(x[:, b], oracle_mod.xray_bin(gaunt_table, rho, u, xe, Z, dist,
                                                      float(e[b]), float(w[b])))
