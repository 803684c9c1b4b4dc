"""Tables of few tiles split a tile's serial work among its threads (the samples
of single and multiple scattering, the theta rows of density): sizes on both
sides of the lines where the shares change, step counts that the shares do not
divide, against the FP64 oracle."""
import numpy as np
import pytest

from fuzzyblue_gb300.params import PRECISION_MIXED, smoke_parameters
from tests.errors import summary

pytestmark = pytest.mark.gpu

# mu_s, nu, mu, r, samples of single and multiple scattering
SIZES = [
    (8, 2, 32, 2, 50),    # 64 rows of 16 texels: eight shares of 51 samples
    (8, 2, 32, 2, 3),     # fewer samples than shares
    (5, 3, 22, 3, 7),     # rows of 15 texels, a last tile with rows missing
    (16, 4, 152, 4, 20),  # 608 rows of 64 texels: 152 tiles of four rows, the first that are not split
    (16, 4, 150, 4, 20),  # just below it
    (32, 8, 4, 2, 9),     # one row of 256 texels per tile: nothing to share
    (11, 1 + 64 // 11, 16, 2, 1),  # two samples
]


@pytest.mark.parametrize("precision", [0, PRECISION_MIXED])
@pytest.mark.parametrize("mu_s,nu,mu,r,steps", SIZES)
def test_split_tiles_match_fp64(builder, oracle, mu_s, nu, mu, r, steps, precision):
    from fuzzyblue_gb300.api import Atmosphere
    p = smoke_parameters(order=3, precision=precision).replace(
        scattering_mu_s_size=mu_s, scattering_nu_size=nu, scattering_mu_size=mu, scattering_r_size=r,
        single_scattering_steps=steps, multiple_scattering_steps=steps, irradiance_mu_s_size=16, irradiance_r_size=4)
    pend = Atmosphere.build(builder, p)
    pend.wait()
    out = pend.atmosphere().to_host()
    pend.release()
    ref = oracle.precompute(p, dtype=np.float64)
    for k in ("transmittance", "irradiance", "scattering"):
        assert np.isfinite(out[k]).all()
        s = summary(out[k], ref[k])
        if precision == PRECISION_MIXED:
            assert s["max"] <= 1e-3, (k, s)
        else:
            # no farther from FP64 than the reference's own FP32 arithmetic
            r32 = summary(oracle.precompute(p)[k].astype(np.float64), ref[k])
            assert s["max"] <= max(1.1 * r32["max"], 2e-3) and s["rms"] <= max(1.1 * r32["rms"], 1e-4), (k, s, r32)
