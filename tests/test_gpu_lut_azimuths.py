"""Spherical correction on azimuth grids in any order: descending, unsorted, with
repeats, with values whose mirror image 360 - r is not exact in binary, outside
[0, 360].  Every grid direction against the oracle, with the parity bar of test_gpu_lut.

A solve at a low sun on a grid of the same size comes first, so that an entry the
kernel left unwritten would hold a correction far from its own."""
import numpy as np
import pytest

from _helpers import oracle_lut
from test_gpu_lut import _check

pytestmark = pytest.mark.gpu

VZA = np.array([0.0, 33.0, 61.5])
GRIDS = {
    "pair": [359.9, 0.1],
    "repeat": [10.0, 350.0, 10.0],
    "ends": [0.0, 360.0, 0.0, 360.0],
    "quadrants": [0.0, 90.0, 180.0, 270.0, 360.0, 90.0],
    "descending": list(np.arange(100)[::-1] * 3.6),
    "descending_fine": list(np.arange(0, 1801, 9)[::-1] * 0.2),
    "unsorted": list(np.random.default_rng(5).permutation(np.arange(144) * 2.5)),
    "outside": [370.0, -10.0, 10.0, 350.0, -350.0, 730.0],
}


@pytest.mark.parametrize("name", GRIDS)
def test_lut_azimuths_in_any_order(gpu, oracle, name):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    raa = np.array(GRIDS[name], dtype=np.float64)
    o = A.default_opts(n_mu=8, n_layers=20, fourier_m_max=4, max_orders=200, pssa=1)
    aer = A.AerosolHolder(0.2, 0.92, *hg_aerosol_moments(0.72, 20))
    kw = dict(surface="black_fresnel_ocean", wind_speed=6.0, raa_deg=0.0)
    low = A.default_case(sza_deg=86.0, vza_deg=80.0, **kw)
    gpu.solve_case_lut(low, o, aer, A.LutHolder(VZA + 25.0, np.linspace(0.0, 360.0, raa.size)))
    c = A.default_case(sza_deg=30.0, vza_deg=0.0, **kw)
    lut = A.LutHolder(VZA, raa)
    gpu.solve_case_lut(c, o, aer, lut)
    _check(lut.out, oracle_lut(oracle, c, o, aer, VZA, raa).out, name)
