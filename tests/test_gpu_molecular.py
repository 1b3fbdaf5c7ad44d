"""The CUDA-core passes at both tile heights of the molecular source (8 levels for
few tasks, 32 for many), with and without aerosol (whose contraction is skipped):
a pixel alone and inside a batch that takes the other height has the same sums in
the same order, so they agree to FP64 rounding of the outputs, and the pixel is at
the parity bar of the oracle."""
import numpy as np
import pytest

from _helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,layers", [(20, 80), (31, 33), (48, 7)])
@pytest.mark.parametrize("tau", [0.0, 0.2])
def test_molecular_tiles(gpu, oracle, monkeypatch, N, layers, tau):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    monkeypatch.setenv("OCRT_GB_SCAN", "column")
    n = 30 if layers > 60 else 250
    c = [A.default_case(surface="black_fresnel_ocean", sza_deg=35.0, vza_deg=20.0, raa_deg=60.0, wind_speed=5.0,
                        wavelength_nm=443.0)] * n
    o = A.default_opts(n_mu=N, n_layers=layers, fourier_m_max=2, max_orders=200)
    a = [A.AerosolHolder(tau, 0.95, *hg_aerosol_moments(0.7, 12))] * n
    one, many = gpu.solve_batch(c[:1], o, a[:1]), gpu.solve_batch(c, o, a)
    for k in ("rho_I", "rho_Q", "rho_U"):
        np.testing.assert_allclose(many[k][[0, n // 2, n - 1]], one[k][0], rtol=1e-12, atol=0)
    assert_parity({k: one[k][0] for k in ("rho_I", "rho_Q", "rho_U")}, oracle.solve(c[0], o, a[0]), f"N={N}")
