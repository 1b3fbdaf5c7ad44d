"""Gradients above 36 streams, where the tensor-map scan of the adjoint does not fit and
its per-column scan runs: against FP64 finite differences of the oracle (the bound of
test_gpu_adjoint), on a batch that mixes them with fewer streams."""
import numpy as np
import pytest

from test_gpu_adjoint import _case, _check_grad, _fd_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mu", [36, 40, 48, 64])
@pytest.mark.parametrize("surface", ["black", "black_fresnel_ocean"])
def test_gradients_above_36_streams(gpu, oracle, n_mu, surface):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    rough = surface != "black"
    c = _case(A, surface, sza_deg=40.0, vza_deg=30.0, raa_deg=60.0)
    kw = dict(n_layers=4, fourier_m_max=2)
    o = A.default_opts(n_mu=n_mu, max_orders=400, tolerance=1e-9, **kw)
    small = A.default_opts(n_mu=16, max_orders=400, tolerance=1e-9, **kw)
    aer = A.AerosolHolder(0.1, 0.93, *hg_aerosol_moments(0.6, 20))
    cot = np.array([1.0, -0.4, 0.3])
    _, g = gpu.solve_batch_adjoint([c, c], [small, o], [aer, aer], None, np.broadcast_to(cot, (2, 1, 3)).copy())
    o_fd = A.default_opts(n_mu=n_mu, max_orders=60, tolerance=1e-300, **kw)
    dt, ss = oracle.layer_defaults(c, o, aer)
    fd_t, fd_s, fd_w = _fd_all(oracle, c, o_fd, aer, dt, ss, cot, rough)
    _check_grad(g["d_dtau"][1, 0], fd_t, "d/ddtau")
    _check_grad(g["d_ssa"][1, 0], fd_s, "d/dssa")
    if rough:
        _check_grad(g["d_wind"][1, 0], fd_w, "d/dwind")
