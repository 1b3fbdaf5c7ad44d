"""Blocks of pairs per CTA of the tensor-core Cox-Munk projection: one pixel (a CTA
per block) and a batch large enough for several blocks a CTA, the last of them
partly filled, give the same solve; and one is at the parity bar of the oracle.
The accumulators of a pair see the same operands in the same order either way, so
pixels agree to FP64 rounding of the outputs."""
import numpy as np
import pytest

from _helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,m_max,n", [(8, 7, 500), (24, 16, 120), (32, 32, 48), (16, 40, 200)])
def test_coxmunk_blocks(gpu, oracle, N, m_max, n):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    c = [A.default_case(surface="black_fresnel_ocean", sza_deg=40.0, vza_deg=25.0, raa_deg=70.0, wind_speed=6.0,
                        wavelength_nm=555.0)] * n
    o = A.default_opts(n_mu=N, n_layers=10, fourier_m_max=m_max, max_orders=100)
    a = [A.AerosolHolder(0.1, 0.95, *hg_aerosol_moments(0.7, 50))] * n
    one, many = gpu.solve_batch(c[:1], o, a[:1]), gpu.solve_batch(c, o, a)
    for k in ("rho_I", "rho_Q", "rho_U"):
        np.testing.assert_allclose(many[k][[0, n // 2, n - 1]], one[k][0], rtol=1e-12, atol=0)
    assert_parity({k: one[k][0] for k in ("rho_I", "rho_Q", "rho_U")}, oracle.solve(c[0], o, a[0]), f"N={N}")
