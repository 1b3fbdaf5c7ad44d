"""Launch shapes are kept per kind of work: k_tables writes the order kernel's parity
operator or the plain one of the separate passes, and a group of either kind is timed
for itself, whichever came first, without a change of results."""
import numpy as np
import pytest

from test_gpu_batch import _batch
from test_gpu_graph import _env

pytestmark = pytest.mark.gpu


def test_tables_are_timed_for_each_form(gpu):
    # a shape that no other test has: modes 0..4 of an expansion to degree 23
    cs, os_, aa = _batch(5, seed=61, n_mu=12, m_max=4, L=23)

    def records():
        return [r for r in gpu.autotune_summary() if r["kernel"] == "k_tables" and list(r["key"])[:3] == [12, 23, 4]]

    assert not records()
    with _env(OCRT_GB_TABLES="simt"):
        r0 = gpu.solve_batch(cs, os_, aa)
    assert len(records()) == 1
    with _env(OCRT_GB_TABLES="simt", OCRT_GB_SCAN="quad"):
        r1 = gpu.solve_batch(cs, os_, aa)
    assert len(records()) == 2
    with _env(OCRT_GB_TABLES="simt"):
        assert np.array_equal(gpu.solve_batch(cs, os_, aa), r0)
    assert len(records()) == 2
    np.testing.assert_allclose(r1["rho_I"], r0["rho_I"], rtol=1e-5)
