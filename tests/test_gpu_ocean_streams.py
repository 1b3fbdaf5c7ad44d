"""The coupled solve on a caller's stream: its inputs are uploaded on the library's
stream, pass by pass, and each pass must find them there.  The result is that of the
library's stream, call after call."""
import ctypes as C

import numpy as np
import pytest

from _helpers import load_golden_ocean, ocean_inputs_from_spec

pytestmark = pytest.mark.gpu


def test_coupled_solve_on_a_callers_stream(gpu):
    torch = pytest.importorskip("torch")
    from ocrt_gb300 import _abi as A
    ins = [ocean_inputs_from_spec(s, n_mu_water=16) for s in load_golden_ocean()["cases"][:3]]
    cs, os_, oc = ([x[k] for x in ins] for k in range(3))
    ref = gpu.solve_batch_ocean(cs, os_, oc)
    n = len(cs)
    ca, oa, oca = (A.Case * n)(*cs), (A.Opts * n)(*os_), (A.Ocean * n)(*[o.struct for o in oc])
    s = torch.cuda.Stream()
    for _ in range(8):
        r, w = (A.Result * n)(), (A.OceanResult * n)()
        assert gpu.lib().ocrt_gb_solve_batch_ocean(n, ca, oa, 1, None, 0, oca, 1, r, w, C.c_void_p(s.cuda_stream)) == 0
        for i in range(n):
            got = {**A.result_dict(r[i]), **A.ocean_result_dict(w[i])}
            assert all(np.array_equal(got[k], ref[i][k]) for k in got), i
