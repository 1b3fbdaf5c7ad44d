"""Level altitudes and layer fractions (k_levels) against the oracle's bisection,
at the edges of its blocks of 63 levels and its range, for both molecular
profiles, with and without an aerosol (down to a trace of either constituent).

The column above an altitude is evaluated to a few 1e-15 of itself, which over a
scale height of 8 km leaves altitudes uncertain by ~1e-13 km and, through the
difference over a layer (1/1024 of the column at least), fractions by ~1e-11;
the bounds leave a factor 100."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 61, 62, 63, 64, 125, 126, 127, 400, 1024])
@pytest.mark.parametrize("profile", [0, 1])
def test_levels_match_oracle(gpu, oracle, layers, profile):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    mom = hg_aerosol_moments(0.7, 8)
    c = A.default_case(sza_deg=30.0, vza_deg=20.0, wavelength_nm=443.0)
    for tau, h in ((None, None), (0.2, 2.0), (1e-4, 0.5), (3.0, 8.0)):
        o = A.default_opts(n_mu=8, n_layers=layers, fourier_m_max=0, rayleigh_profile=profile,
                           **({} if h is None else {"aer_h_km": h}))
        aer = None if tau is None else A.AerosolHolder(tau, 0.9, *mom)
        z, zr = gpu.layer_gas(c, o, aer)[1], oracle.layer_gas(c, o, aer)[1]
        np.testing.assert_allclose(z, zr, rtol=0, atol=1e-11)
        (dt, w), (dtr, wr) = gpu.layer_defaults(c, o, aer), oracle.layer_defaults(c, o, aer)
        np.testing.assert_allclose(dt, dtr, rtol=1e-12, atol=0)
        np.testing.assert_allclose(w, wr, rtol=0, atol=1e-9)
