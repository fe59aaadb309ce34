"""GPU parity of the per-cell quantities where their kernels change path: cells
and energies outside the plain range of the hoisted emission (temperatures at
the edges of and beyond the Gaunt table, zero, negative and non-finite inputs,
results that underflow), cell counts around a warp and a block, bin counts
around the warp and the bin chunk. Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import same_bits

pytestmark = pytest.mark.gpu

Z, DL = 0.2, 978500.0
X0, DX = 0.105322271585, 0.010644


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    # internal energies from far below to far above the table's temperatures
    u = np.exp(rng.uniform(np.log(1e-8), np.log(1e22), n)).astype(np.float32)
    rho = np.exp(rng.uniform(np.log(1e-12), np.log(1e9), n)).astype(np.float32)
    xe = rng.uniform(0.0, 2.0, n).astype(np.float32)
    u[::2] = np.exp(rng.uniform(np.log(1e3), np.log(3e6), len(u[::2])))  # the usual range
    special = [0.0, -1.0, np.nan, np.inf, 1e-45, 1e-38, 3e38, -np.inf]
    k = min(n, len(special))
    for a in (u, rho, xe):
        at = rng.permutation(n)[:k]
        a[at] = np.float32(special)[rng.permutation(len(special))[:k]]
    return rho, u, xe


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 5000])
def test_quantities_edge_cells(ctx, oracle_mod, gaunt_table, n):
    from illcrawl_b200 import synthetic
    ctx.load_gaunt()
    arf = synthetic.synthetic_arf(n=130)
    ctx.load_arf(arf, X0, DX)
    rho, u, xe = _inputs(n, 60 + n)
    for lo, hi, ns in ((0.5, 7.0, 100), (0.1, 10.0, 7)):
        assert same_bits(ctx.xray_flux(rho, u, xe, Z, DL, lo, hi, ns),
                         oracle_mod.xray_band(gaunt_table, rho, u, xe, Z, DL, lo, hi, ns))
        assert same_bits(ctx.xray_photon_flux(rho, u, xe, Z, DL, lo, hi, ns),
                         oracle_mod.xray_photon_flux(gaunt_table, rho, u, xe, Z, DL, lo, hi, ns))
    assert same_bits(ctx.chandra_count_rate(rho, u, xe, Z, DL),
                     oracle_mod.chandra_count_rate(gaunt_table, arf, X0, DX, rho, u, xe, Z, DL))
    # a luminosity distance and energies beyond the plain range
    for dist in (1e-9, 3e9):
        assert same_bits(ctx.xray_spectral_flux(rho, u, xe, 1.0, 0.1, Z, dist),
                         oracle_mod.xray_bin(gaunt_table, rho, u, xe, Z, dist, 1.0, 0.1))
    for e in (0.0, 1e-14, 1e-6, 30.0, 1e13):
        assert same_bits(ctx.xray_spectral_flux(rho, u, xe, e, 0.1, Z, DL),
                         oracle_mod.xray_bin(gaunt_table, rho, u, xe, Z, DL, e, 0.1))
        assert same_bits(
            ctx.chandra_spectral_count_rate(rho, u, xe, e, 0.1, Z, DL),
            oracle_mod.chandra_spectral_count_rate(gaunt_table, arf, X0, DX, rho, u, xe, Z, DL, e,
                                                   0.1))


@pytest.mark.parametrize("n_bins", [1, 2, 31, 32, 33, 127, 128, 129, 300])
def test_bin_tables(ctx, oracle_mod, gaunt_table, n_bins):
    from illcrawl_b200 import synthetic
    ctx.load_gaunt()
    arf = synthetic.synthetic_arf()
    ctx.load_arf(arf, X0, DX)
    for n in (1, 45, 700):
        rho, u, xe = _inputs(n, n_bins)
        edges = np.geomspace(0.2, 11.0, n_bins + 1)
        e, w = edges[:-1].astype(np.float32), np.diff(edges).astype(np.float32)
        x = ctx.xray_spectrum(rho, u, xe, e, w, Z, DL)
        c = ctx.chandra_spectrum(rho, u, xe, e, w, Z, DL)
        for b in sorted({0, n_bins // 2, n_bins - 1}):
            assert same_bits(x[:, b], oracle_mod.xray_bin(gaunt_table, rho, u, xe, Z, DL,
                                                          float(e[b]), float(w[b])))
            assert same_bits(c[:, b], oracle_mod.chandra_spectral_count_rate(
                gaunt_table, arf, X0, DX, rho, u, xe, Z, DL, float(e[b]), float(w[b])))
        # every bin against the one-bin quantity
        for b in range(n_bins):
            assert same_bits(x[:, b], ctx.xray_spectral_flux(rho, u, xe, float(e[b]), float(w[b]),
                                                             Z, DL))


@pytest.mark.parametrize("shape", [(2, 2), (1, 9), (5000, 2), (2, 5000), (146, 81)])
def test_other_gaunt_tables(ctx, oracle_mod, gaunt_table, shape):
    """Tables of other shapes (rows, columns); the long ones are kept unpadded."""
    rng = np.random.default_rng(7)
    t = rng.uniform(0.5, 2.0, shape).astype(np.float32)
    rho, u, xe = _inputs(600, 8)
    try:
        # the oracle's spacing and origin (gaunt_factor.cpp:30-41)
        ctx.load_gaunt(t)
        assert same_bits(ctx.xray_flux(rho, u, xe, Z, DL, 0.5, 7.0, 100),
                         oracle_mod.xray_band(t, rho, u, xe, Z, DL, 0.5, 7.0, 100))
        assert same_bits(ctx.xray_spectral_flux(rho, u, xe, 2.0, 0.1, Z, DL),
                         oracle_mod.xray_bin(t, rho, u, xe, Z, DL, 2.0, 0.1))
    finally:
        ctx.load_gaunt()
