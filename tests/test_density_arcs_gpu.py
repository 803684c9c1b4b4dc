"""Scattering density of orders >= 3 by arcs (fb_density_arcs.cuh): sizes at
the edges of its tiles (32 mu rows, 8 warps, up to 7 nu texels per warp beside
the two ends) and of the rule that chooses it, against the FP64 oracle."""
import numpy as np
import pytest

from fuzzyblue_gb300.params import PRECISION_MIXED, smoke_parameters
from tests.errors import summary

pytestmark = pytest.mark.gpu

# nu, mu_s, mu, r, density_samples, irradiance mu_s
SIZES = [
    (2, 8, 32, 4, 16, 64),    # the ends only
    (3, 7, 34, 3, 16, 2),     # one texel between the ends, two mu rows in the last tile, no ground knots
    (9, 9, 30, 2, 16, 33),    # as many nu texels as one warp takes
    (10, 5, 66, 2, 16, 512),  # two warps per column; the longest ground row that goes by arcs
    (17, 6, 20, 2, 16, 16),   # three warps per column, two of eight warps idle
    (24, 4, 16, 2, 16, 16),   # near the most knots per row
    (40, 4, 16, 2, 16, 16),   # more knots than the rule takes: the direct sums
    (5, 9, 64, 2, 2, 64),     # the fewest directions
    (6, 11, 18, 3, 32, 64),   # the most
]


@pytest.mark.parametrize("nu,mu_s,mu,r,samples,ir_mus", SIZES)
def test_arcs_match_fp64(builder, oracle, nu, mu_s, mu, r, samples, ir_mus):
    from fuzzyblue_gb300.api import Atmosphere
    p = smoke_parameters(order=3, precision=PRECISION_MIXED).replace(
        scattering_nu_size=nu, scattering_mu_s_size=mu_s, scattering_mu_size=mu, scattering_r_size=r,
        density_samples=samples, irradiance_mu_s_size=ir_mus, irradiance_r_size=4)
    pend = Atmosphere.build(builder, p)
    pend.wait()
    out = pend.atmosphere().to_host()
    inter = {k: v.to_numpy() for k, v in pend.intermediates().items()}
    pend.release()
    o2 = Atmosphere.build(builder, p.replace(order=2))
    o2.wait()
    i2 = {k: v.to_numpy() for k, v in o2.intermediates().items()}
    o2.release()
    f64 = np.float64

    def flat(a):
        return np.ascontiguousarray(a.reshape(-1, 4)).astype(f64)

    # the density of order 3 alone, on the GPU's own order-2 inputs
    nsc = p.texel_counts()[2]
    idx = np.unique(np.random.default_rng(7).choice(nsc, min(nsc, 2048), replace=False)).astype(np.int64)
    ref = oracle.scattering_density(p, 3, flat(out["transmittance"]), flat(i2["delta_rayleigh"]),
                                    flat(i2["delta_mie"]), flat(i2["delta_multiple_scattering"]),
                                    flat(i2["delta_irradiance_1"]), idx=idx, dtype=f64)
    got = inter["scattering_density"].reshape(-1, 4)[idx]
    assert np.isfinite(got).all()
    s = summary(got.astype(f64), ref)
    assert s["max"] <= 1e-3 and s["rms"] <= 1e-4, s
    whole = oracle.precompute(p, dtype=f64)
    for k in ("transmittance", "irradiance", "scattering"):
        assert summary(out[k], whole[k])["max"] <= 1e-3, k
