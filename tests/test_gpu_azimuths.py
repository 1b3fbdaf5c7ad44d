"""Rough surfaces on every kind of Cox-Munk azimuth grid (opts.n_phi_surface): below, at
and above the default 1024, multiples of the tensor-core chunk (64) and others, against
the oracle on the same grid, looking into and away from the sun glint.  A batch that
mixes grids gives each pixel its own."""
import numpy as np
import pytest

from _helpers import assert_parity

pytestmark = pytest.mark.gpu

NPHI = [64, 100, 128, 250, 256, 512, 960, 1024, 1030, 2048, 4096]


def _case(A, raa, wind=4.0):
    return A.default_case(surface="black_fresnel_ocean", sza_deg=40.0, vza_deg=35.0, raa_deg=raa, wind_speed=wind,
                          wavelength_nm=555.0)


@pytest.mark.parametrize("nphi", NPHI)
@pytest.mark.parametrize("n_mu, m_max", [(8, 4), (16, 12), (31, 70)])
def test_azimuth_grids_match_oracle(gpu, oracle, nphi, n_mu, m_max):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    aer = A.AerosolHolder(0.1, 0.95, *hg_aerosol_moments(0.6, 15))
    o = A.default_opts(n_mu=n_mu, n_layers=6, fourier_m_max=m_max, n_phi_surface=nphi, max_orders=100, tolerance=1e-8)
    for raa in (5.0, 175.0):
        c = _case(A, raa)
        assert_parity(gpu.solve_case(c, o, aer), oracle.solve(c, o, aer), f"nphi {nphi} raa {raa}")


def test_mixed_grids_in_a_batch(gpu, oracle):
    from ocrt_gb300 import _abi as A
    cs = [_case(A, 170.0, 3.0 + i) for i in range(len(NPHI))]
    os_ = [A.default_opts(n_mu=12, n_layers=8, fourier_m_max=6, n_phi_surface=n, max_orders=100) for n in NPHI]
    res = gpu.solve_batch(cs, os_, None)
    for i, (c, o) in enumerate(zip(cs, os_)):
        assert_parity({k: float(res[k][i]) for k in ("rho_I", "rho_Q", "rho_U")}, oracle.solve(c, o), f"nphi {NPHI[i]}")


@pytest.mark.parametrize("nphi", [128, 256, 500])
def test_wind_gradient_on_small_grids(gpu, oracle, nphi):
    from ocrt_gb300 import _abi as A
    from _helpers import fd_gradient
    c = _case(A, 165.0)
    o = A.default_opts(n_mu=8, n_layers=4, fourier_m_max=4, n_phi_surface=nphi, max_orders=300, tolerance=1e-9)
    cot = np.array([1.0, 0.0, 0.0])
    _, g = gpu.solve_batch_adjoint([c], o, None, None, cot[None, None, :])
    o_fd = A.default_opts(n_mu=8, n_layers=4, fourier_m_max=4, n_phi_surface=nphi, max_orders=60, tolerance=1e-300)
    dt, ss = oracle.layer_defaults(c, o, None)
    fd = fd_gradient(oracle, c, o_fd, None, dt, ss, cot, [("wind", None)])[0]
    assert abs(g["d_wind"][0, 0] - fd) <= 1e-4 * abs(fd) + 1e-8
