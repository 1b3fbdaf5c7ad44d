"""All orders of a task in one CTA (k_orders: N = 8, 16, 24, 32, forward solves)
at the edges of its shape: tiles of 112 levels (one tile, a tile of one level,
two, three and four tiles, so kept, spilled and reloaded ones), groups of 16
levels, the smallest column, every surface, layers of unequal optical depth,
molecules alone, the view as an inserted slot and as a Gauss node.

Against the FP64 oracle at the parity bar, and against the separate passes
(OCRT_GB_SOURCE_KERNEL=simt) at 1e-5 relative in I and 1e-6 absolute in Q and U:
an order is an FP32 recurrence over at most 400 levels, about sqrt(400) x 6e-8
= 1.2e-6 of the field per path, the operators differ by the same FP32 rounding,
and a mode may stop one order earlier (tolerance 1e-7)."""
import numpy as np
import pytest

from _helpers import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 14, 111, 112, 128, 223, 224, 336, 400])
@pytest.mark.parametrize("N", [8, 16, 24, 32])
def test_orders_match_oracle_and_separate_passes(gpu, oracle, monkeypatch, N, layers):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    rng = np.random.default_rng(1000 * N + layers)
    mom = hg_aerosol_moments(0.7, 40)
    cases, aers, ly = [], [], []
    for surface, aerosol, uneven in (("black_fresnel_ocean", True, False), ("black", True, True), ("flat", False, False),
                                     ("black_fresnel_ocean", False, True)):
        cases.append(A.default_case(surface=surface, sza_deg=rng.uniform(5, 70), vza_deg=rng.uniform(0, 60),
                                    raa_deg=rng.uniform(0, 180), wind_speed=rng.uniform(1, 10),
                                    wavelength_nm=float(rng.choice([443.0, 865.0]))))
        aers.append(A.AerosolHolder(rng.uniform(0.05, 0.4) if aerosol else 0.0, rng.uniform(0.85, 0.99), *mom))
        dt = rng.uniform(0.5, 1.5, layers) * 0.3 / layers if uneven else None
        ly.append(A.LayersHolder(layers, dt, None))
    o = A.default_opts(n_mu=N, n_layers=layers, fourier_m_max=4, max_orders=300, tolerance=1e-7,
                       view_as_node=int(layers % 2))
    monkeypatch.delenv("OCRT_GB_SOURCE_KERNEL", raising=False)
    got, _ = gpu.solve_batch_adjoint(cases, o, aers, ly, None)
    monkeypatch.setenv("OCRT_GB_SOURCE_KERNEL", "simt")
    sep, _ = gpu.solve_batch_adjoint(cases, o, aers, ly, None)
    np.testing.assert_allclose(got["rho_I"], sep["rho_I"], rtol=1e-5, atol=0)
    for k in ("rho_Q", "rho_U"):
        np.testing.assert_allclose(got[k], sep[k], rtol=0, atol=1e-6)
    for i, c in enumerate(cases):
        ref = oracle.solve_layers(c, o, aers[i], ly[i].dtau, None)
        assert_parity({k: got[k][i] for k in ("rho_I", "rho_Q", "rho_U")}, ref, f"N={N} layers={layers} pixel {i}")


@pytest.mark.parametrize("layers", [2, 7, 8, 112, 113, 226])
@pytest.mark.parametrize("max_orders", [1, 2])
def test_first_order(gpu, oracle, monkeypatch, max_orders, layers):
    """Order 1 inside the kernel (eight levels at a time, and up to four where a
    column starts, ends or is not plain): tasks that end with it or go one order
    on, every surface over even and uneven layers, same bounds."""
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    rng = np.random.default_rng(layers)
    mom = hg_aerosol_moments(0.7, 40)
    cases, ly = [], []
    for i, surface in enumerate(("black_fresnel_ocean", "black", "flat") * 2):
        cases.append(A.default_case(surface=surface, sza_deg=rng.uniform(5, 70), vza_deg=rng.uniform(0, 60),
                                    raa_deg=rng.uniform(0, 180), wind_speed=rng.uniform(1, 10), wavelength_nm=555.0))
        dt = rng.uniform(0.5, 1.5, layers) * 0.3 / layers if i >= 3 else None
        ly.append(A.LayersHolder(layers, dt, None))
    aer = A.AerosolHolder(0.2, 0.95, *mom)
    o = A.default_opts(n_mu=24, n_layers=layers, fourier_m_max=3, max_orders=max_orders, tolerance=1e-7)
    monkeypatch.delenv("OCRT_GB_SOURCE_KERNEL", raising=False)
    got, _ = gpu.solve_batch_adjoint(cases, o, [aer] * 6, ly, None)
    monkeypatch.setenv("OCRT_GB_SOURCE_KERNEL", "simt")
    sep, _ = gpu.solve_batch_adjoint(cases, o, [aer] * 6, ly, None)
    np.testing.assert_allclose(got["rho_I"], sep["rho_I"], rtol=1e-5, atol=0)
    for k in ("rho_Q", "rho_U"):
        np.testing.assert_allclose(got[k], sep[k], rtol=0, atol=1e-6)
    for i, c in enumerate(cases):
        ref = oracle.solve_layers(c, o, aer, ly[i].dtau, None)
        assert_parity({k: got[k][i] for k in ("rho_I", "rho_Q", "rho_U")}, ref, f"layers={layers} pixel {i}")


@pytest.mark.parametrize("N,layers,max_orders,van", [(8, 2, 300, 1), (8, 15, 1, 1), (16, 16, 2, 0), (24, 17, 300, 1),
                                                     (32, 31, 2, 1), (16, 111, 300, 1), (24, 112, 300, 0),
                                                     (32, 225, 300, 1), (8, 337, 300, 1)])
def test_adjoint_orders_match_separate_passes(gpu, monkeypatch, N, layers, max_orders, van):
    """The adjoint's orders in one CTA against the separate transposed passes, at
    the edges of groups, tiles and order counts, more (task, row) items than the
    chip has SMs (a zero output row among them), even and uneven layers, the view
    inserted, between nodes and on a node.  Both run in FP32 on the same linear
    system, so gradients agree to 1e-5 of the largest of their group (the order
    sums' rounding, sqrt(337) x 6e-8, and a last order of 1e-7)."""
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    rng = np.random.default_rng(100 * N + layers)
    gmu = np.polynomial.legendre.leggauss(2 * N)[0][N:]
    n = 24
    cases, aers, ly = [], [], []
    for i in range(n):
        vza = np.degrees(np.arccos(gmu[N // 2])) if i == 5 else rng.uniform(0, 60)
        cases.append(A.default_case(surface=["black", "black_fresnel_ocean"][i % 2], sza_deg=rng.uniform(5, 70),
                                    vza_deg=vza, raa_deg=rng.uniform(0, 180), wind_speed=rng.uniform(1, 10),
                                    wavelength_nm=555.0))
        aers.append(A.AerosolHolder(rng.uniform(0.05, 0.4), 0.95, *hg_aerosol_moments(0.7, 24)))
        dt = rng.uniform(0.5, 1.5, layers) * 0.3 / layers if i % 3 == 0 else None
        ly.append(A.LayersHolder(layers, dt, None))
    o = A.default_opts(n_mu=N, n_layers=layers, fourier_m_max=3, max_orders=max_orders, tolerance=1e-7,
                       view_as_node=van)
    cot = np.broadcast_to(np.eye(3), (n, 3, 3)).copy()
    cot[1, 0] = 0.0
    monkeypatch.delenv("OCRT_GB_SOURCE_KERNEL", raising=False)
    r1, g1 = gpu.solve_batch_adjoint(cases, o, aers, ly, cot)
    monkeypatch.setenv("OCRT_GB_SOURCE_KERNEL", "simt")
    r2, g2 = gpu.solve_batch_adjoint(cases, o, aers, ly, cot)
    np.testing.assert_allclose(r1["rho_I"], r2["rho_I"], rtol=1e-5)
    for k in ("d_dtau", "d_ssa", "d_wind"):
        for i in range(n):
            scale = np.abs(g2[k][i]).max()
            assert np.abs(g1[k][i] - g2[k][i]).max() <= 1e-5 * scale + 1e-12, (k, i)


@pytest.mark.parametrize("layers", [14, 113])
@pytest.mark.parametrize("N", [12, 28])
def test_orders_at_multiples_of_four(gpu, oracle, monkeypatch, N, layers):
    """Stream counts that fill neither a 16-deep MMA step nor the boundary sum's
    steps of 8 slots: forward and adjoint, same bounds."""
    test_orders_match_oracle_and_separate_passes(gpu, oracle, monkeypatch, N, layers)
    test_adjoint_orders_match_separate_passes(gpu, monkeypatch, N, layers, 300, layers % 2)
