"""Bias of the order kernel's products against FP32 ones.

The tensor cores' accumulator truncates at every step.  With the incoming intensity
last, a sum is at its full size for the last products of two 16-column steps only; each
loses less than an ulp, 2^-23 of the value, so a source is low by less than 2^-22, and
so is, in the mean over pixels, the part of a reflectance that came of it, against
CUDA-core products rounded to nearest.  (With the intensity first a sum took 24
truncating steps at full size.)"""
import numpy as np
import pytest

from test_gpu_graph import _env

pytestmark = pytest.mark.gpu


def _pixels(A, n_mu, n=96):
    from synthetic import hg_aerosol_moments
    rng = np.random.default_rng(33)
    out = []
    for i in range(n):
        c = A.default_case(surface=("black_fresnel_ocean", "black", "black_fresnel_ocean", "flat")[i % 4],
                           sza_deg=rng.uniform(5, 70), vza_deg=rng.uniform(0, 60), raa_deg=rng.uniform(0, 180),
                           wind_speed=rng.uniform(1, 10), wavelength_nm=float(rng.choice([443.0, 555.0, 865.0])))
        o = A.default_opts(n_mu=n_mu, n_layers=int(rng.choice([20, 60, 150])), fourier_m_max=int(rng.choice([2, 6, 12])),
                           max_orders=500, tolerance=1e-7, pssa=0)
        a = A.AerosolHolder(rng.uniform(0.02, 0.5), rng.uniform(0.8, 1.0), *hg_aerosol_moments(rng.uniform(0.5, 0.8), 60))
        out.append((c, o, None if i % 6 == 5 else a))
    return out


@pytest.mark.parametrize("n_mu", [24, 28])
def test_products_lose_less_than_two_ulps(gpu, n_mu):
    from ocrt_gb300 import _abi as A
    pix = _pixels(A, n_mu)
    one = np.array([gpu.solve_case(*p)["rho_I"] for p in pix])
    with _env(OCRT_GB_SOURCE_KERNEL="simt"):
        simt = np.array([gpu.solve_case(*p)["rho_I"] for p in pix])
    bias = np.mean((one - simt) / simt)
    print(f"mean bias {bias:+.2e}")
    assert abs(bias) <= 2.0 ** -22
