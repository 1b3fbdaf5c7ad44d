"""Work that the order kernel is credited with: in the parity form the contraction takes
36 N^2 multiply-adds' worth of FLOPs a level and order (half of the dense 72 N^2) and the
recurrences 30 N a layer and order; bytes are those of the operator, the surface rows and
the totals at the two output levels, whatever the number of orders."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mu, layers, surface", [(8, 20, "black"), (24, 40, "black_fresnel_ocean")])
def test_order_kernel_work(gpu, n_mu, layers, surface):
    from ocrt_gb300 import _abi as A
    c = A.default_case(surface=surface, wind_speed=5.0, sza_deg=40.0, vza_deg=20.0)
    o = A.default_opts(n_mu=n_mu, n_layers=layers, fourier_m_max=0, pssa=0)
    plan = gpu.Plan([c], [o], None)
    plan.execute()
    orders = int(plan.results()["order_modes"][0])
    ks = plan.kernel_stats()["source_gemm_tcgen05"]
    plan.close()
    N, K, NR = n_mu, layers + 1, n_mu + 1
    assert orders > 2
    assert ks["flops"] == (orders - 1) * 36.0 * N * N * K + orders * 30.0 * N * layers
    rows = (3 * NR + 3 + 7) // 8 * 8
    srf = 3 * N * ((3 * NR + 31) // 32 * 32) * 4 if surface != "black" else 0
    assert ks["bytes"] == 9 * rows * 128 + srf + 2 * 6 * NR * 4
