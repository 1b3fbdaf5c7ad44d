"""An execute under a caller's capture (a plan of order 1 only, whose eager execute
polls nothing) keeps to the caller's stream: the library's second stream stays free, so
that another plan can execute while the caller is still capturing."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_batch import _batch
from test_gpu_graph import _env

pytestmark = pytest.mark.gpu


def test_another_plan_executes_while_a_caller_captures(gpu):
    torch = pytest.importorskip("torch")
    cs, os_, aa = _batch(5, seed=71, n_mu=16, m_max=4)
    for o in os_:
        o.max_orders = 1
    other = _batch(7, seed=72, n_mu=16, m_max=3)
    s = [torch.cuda.Stream() for _ in range(2)]
    sp = [C.c_void_p(x.cuda_stream) for x in s]
    with _env(OCRT_GB_GRAPH="0"):
        p0, p1 = gpu.Plan(cs, os_, aa), gpu.Plan(*other)
        p0.execute(sp[0])
        r0 = p0.results(sp[0])
        p1.execute(sp[1])
        r1 = p1.results(sp[1])
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s[0], capture_error_mode="relaxed"):
            p0.execute(sp[0])
            p1.execute(sp[1])
        for _ in range(2):
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(p0.results(sp[0]), r0)
        assert np.array_equal(p1.results(sp[1]), r1)
        del g
        p0.close()
        p1.close()
