"""The allocation-free solve at the smallest stream counts, where the molecular factor is
larger than the plain operator: against the oracle and the allocating solve."""
import pytest

from _helpers import assert_parity
from test_zz_no_alloc import _call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mu", [2, 3, 4, 5])
@pytest.mark.parametrize("surface", ["black", "flat", "black_fresnel_ocean"])
def test_noalloc_at_few_streams(gpu, oracle, n_mu, surface):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    aer = A.AerosolHolder(0.2, 0.9, *hg_aerosol_moments(0.3, 2))
    c = A.default_case(surface=surface, sza_deg=40.0, vza_deg=25.0, raa_deg=60.0, wind_speed=5.0)
    for m_max, a in ((2, None), (2, aer), (5, aer)):
        o = A.default_opts(n_mu=n_mu, n_layers=10, fourier_m_max=m_max, max_orders=200, tolerance=1e-8)
        rc, got = _call(gpu, c, o, a)
        assert rc == 0
        assert_parity(got, oracle.solve(c, o, a), f"N={n_mu} {surface} vs the oracle")
        assert_parity(got, gpu.solve_case(c, o, a), f"N={n_mu} {surface} vs solve_case")
