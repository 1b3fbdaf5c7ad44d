"""A plan's work and its buffers on callers' streams.  An execute returns with its work
queued; results and gradients on another stream, a later execute on another stream and
destroying the plan wait for it, and two plans on two streams, which share the library's
second stream, do not disturb each other.

The executes are queued behind some 20 ms of waiting, so that what does not wait finds
the buffers as they were before."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_batch import _batch

pytestmark = pytest.mark.gpu

DELAY = 40_000_000          # clock cycles of torch.cuda._sleep


@pytest.fixture
def streams():
    torch = pytest.importorskip("torch")
    s = [torch.cuda.Stream() for _ in range(2)]

    def behind(i):
        with torch.cuda.stream(s[i]):
            torch.cuda._sleep(DELAY)
        return C.c_void_p(s[i].cuda_stream)

    yield s, behind
    torch.cuda.synchronize()


def _ref(gpu, cs, os_, aa):
    p = gpu.Plan(cs, os_, aa)
    p.execute()
    r = p.results()
    p.close()
    return r


@pytest.mark.parametrize("n_mu", [16, 20])
def test_results_wait_for_an_execute_on_another_stream(gpu, streams, n_mu):
    s, behind = streams
    cs, os_, aa = _batch(6, seed=51, n_mu=n_mu, m_max=3)
    ref = _ref(gpu, cs, os_, aa)
    plan = gpu.Plan(cs, os_, aa)
    for other in (None, C.c_void_p(s[1].cuda_stream)):
        plan.execute(behind(0))
        assert np.array_equal(plan.results(other), ref)
    plan.execute()                                  # library's stream, results on a caller's
    assert np.array_equal(plan.results(C.c_void_p(s[0].cuda_stream)), ref)
    plan.close()


def test_execute_waits_for_the_one_before(gpu, streams):
    s, behind = streams
    cs, os_, aa = _batch(24, seed=52, n_mu=16, m_max=6)
    ref = _ref(gpu, cs, os_, aa)
    plan = gpu.Plan(cs, os_, aa)
    plan.execute(behind(0))
    plan.execute(C.c_void_p(s[1].cuda_stream))      # would overlap the first in the same buffers
    plan.execute()
    plan.execute(C.c_void_p(s[1].cuda_stream))
    assert np.array_equal(plan.results(C.c_void_p(s[1].cuda_stream)), ref)
    plan.close()


def test_gradients_wait(gpu, streams):
    from ocrt_gb300 import _abi as A
    from synthetic import hg_aerosol_moments
    s, behind = streams
    c = [A.default_case(surface="black_fresnel_ocean", wind_speed=5.0, sza_deg=35.0, vza_deg=25.0, raa_deg=70.0)]
    o = A.default_opts(n_mu=8, n_layers=12, fourier_m_max=3, max_orders=200)
    a = [A.AerosolHolder(0.1, 0.93, *hg_aerosol_moments(0.7, 20))]
    cot = np.eye(3)[None].copy()
    p = gpu.Plan(c, o, a, cot=cot)
    p.execute()
    ref = p.gradients()
    p.close()
    plan = gpu.Plan(c, o, a, cot=cot)
    plan.execute(behind(0))
    g = plan.gradients()
    for k in ("d_dtau", "d_ssa", "d_wind"):
        assert np.array_equal(g[k], ref[k]), k
    plan.close()


def test_close_waits(gpu, streams):
    s, behind = streams
    cs, os_, aa = _batch(6, seed=53, n_mu=16, m_max=3)
    plan = gpu.Plan(cs, os_, aa)
    plan.execute(behind(0))
    plan.close()
    assert s[0].query()                             # nothing of it is still to run


def test_two_plans_on_two_streams(gpu, streams):
    s, behind = streams
    sets = [_batch(12, seed=54, n_mu=16, m_max=5), _batch(9, seed=55, n_mu=24, m_max=4)]
    refs = [_ref(gpu, *b) for b in sets]
    plans = [gpu.Plan(*b) for b in sets]
    sp = [behind(0), behind(1)]
    for _ in range(4):                              # eager, captured, replayed
        for p, x in zip(plans, sp):
            p.execute(x)
        for p, x, r in zip(plans, sp, refs):
            assert np.array_equal(p.results(x), r)
    for p in plans:
        p.close()
