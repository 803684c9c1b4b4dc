"""Density at the sizes where its tables nearly fill an SM's shared memory: tiles
of many columns and few mu rows, few nu slices, and the longest ground rows
beside many density samples or nu slices (limit_density_shape, fb_capi.cu)."""
import numpy as np
import pytest

from fuzzyblue_gb300.params import PRECISION_MIXED, PRECISION_PLAIN, smoke_parameters
from tests.errors import summary

pytestmark = pytest.mark.gpu

# nu, mu_s, mu, r, density_samples, irradiance mu_s, precision, order
SIZES = [
    (2, 64, 4, 64, 16, 64, PRECISION_MIXED, 2),     # 32 columns of 4 mu rows, 8 records each
    (9, 28, 4, 64, 16, 2048, PRECISION_MIXED, 2),   # 16 records for 8 intervals, a long ground row
    (2, 64, 4, 64, 20, 4096, PRECISION_PLAIN, 3),   # direct sums of order 3
    (50, 2, 18, 2, 32, 4096, PRECISION_PLAIN, 2),   # few tiles, no room for split sums
]


@pytest.mark.parametrize("nu,mu_s,mu,r,samples,ir_mus,precision,order", SIZES)
def test_density_at_the_limits(builder, oracle, nu, mu_s, mu, r, samples, ir_mus, precision, order):
    from fuzzyblue_gb300.api import Atmosphere
    p = smoke_parameters(order=order, precision=precision).replace(
        scattering_nu_size=nu, scattering_mu_s_size=mu_s, scattering_mu_size=mu, scattering_r_size=r,
        density_samples=samples, irradiance_mu_s_size=ir_mus, irradiance_r_size=4)

    def build(n):
        pend = Atmosphere.build(builder, p.replace(order=n))
        pend.wait()
        inter = {k: v.to_numpy() for k, v in pend.intermediates().items()}
        transmittance = pend.atmosphere().to_host()["transmittance"]
        pend.release()
        return transmittance, inter

    def flat(a):
        return np.ascontiguousarray(a.reshape(-1, 4))

    transmittance, inter = build(order)
    # the multiple scattering of the order before (order 2 reads single scattering alone)
    multiple = build(order - 1)[1]["delta_multiple_scattering"] if order > 2 else np.zeros_like(
        inter["delta_multiple_scattering"])
    nsc = p.texel_counts()[2]
    idx = np.unique(np.random.default_rng(11).choice(nsc, min(nsc, 1024), replace=False)).astype(np.int64)
    inputs = [flat(a) for a in (transmittance, inter["delta_rayleigh"], inter["delta_mie"], multiple,
                                inter["delta_irradiance_%d" % (order & 1)])]

    def reference(real):
        return oracle.scattering_density(p, order, *(a.astype(real) for a in inputs), idx=idx,
                                         dtype=real).astype(np.float64)

    got = inter["scattering_density"].reshape(-1, 4)[idx]
    assert np.isfinite(got).all()
    exact = reference(np.float64)
    # mixed: the bound of a pass alone; plain: FP32 itself is off where a nu slice's
    # texture coordinate rounds into the one before it (nu not a power of two)
    bound = 1e-3 if precision == PRECISION_MIXED else max(2e-2, 2 * summary(reference(np.float32), exact)["max"])
    s = summary(got.astype(np.float64), exact)
    assert s["max"] <= bound, (s, bound)
