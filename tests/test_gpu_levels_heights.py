"""Level altitudes (k_levels) for scale heights far from the usual ones, which the entry
points take: nearly uniform columns (1e10 km), layers thinner than the FP32 search
resolves (1e-9 km); against the oracle's bisection.

Tolerance.  Column fractions are (exp(-z / h) - e) / (1 - e), e = exp(-100 / h), with
exp good to an ulp: an altitude is uncertain by a few 2.2e-16 times the column's own
scale h (1 - e) at z, and by 2.2e-16 h / (100 / h) km for
large h: 4.4e-6 km at 1e10, taken fourfold; at ordinary heights 1e-11 km as in
test_gpu_levels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ray_h, aer_h, atol", [
    (8.0, 1e10, 2e-5), (1e10, 2.0, 2e-5), (1e10, 1e10, 2e-5), (8.0, 1e8, 2e-7), (1e8, 2.0, 2e-7),
    (8.0, 1e4, 1e-9), (8.0, 1e-4, 1e-11), (8.0, 1e-9, 1e-11)])
def test_levels_at_extreme_scale_heights(gpu, oracle, ray_h, aer_h, atol):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    c = A.default_case(sza_deg=30.0, vza_deg=20.0, wavelength_nm=443.0)
    aer = A.AerosolHolder(0.3, 0.9, *hg_aerosol_moments(0.7, 8))
    o = A.default_opts(n_mu=8, n_layers=41, fourier_m_max=0, rayleigh_profile=1, rayleigh_h_km=ray_h, aer_h_km=aer_h,
                       pssa=0)
    z, zr = gpu.layer_gas(c, o, aer)[1], oracle.layer_gas(c, o, aer)[1]
    np.testing.assert_allclose(z, zr, rtol=0, atol=atol)
