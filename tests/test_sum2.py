"""The two-word FP32 sums of csrc/sum2.cuh, which the water-to-air quadrature keeps its
node and azimuth sums in, compiled for the host and compared with FP64.

Bounds.  A head s and a tail c: every two-sum and FMA product error is exact, so what
is lost is the rounding of c, which never exceeds n 2^-24 of the sum of magnitudes;
each of its n additions rounds by 2^-24 of that: n^2 2^-48 in all.  (Plain FP32
accumulation loses up to n 2^-24 and misses this by far.)  sum2_sqrt: half an ulp and a
part in 2^20 of it for the correction's own rounding."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import ocrt_gb300

CSRC = os.path.join(os.path.dirname(ocrt_gb300.__file__), "csrc")
CODE = """
#include "sum2.cuh"
extern "C" void sums(int n, const float *h, const float *l, const float *t, float *out)
{
    float s = 0.f, c = 0.f;
    for (int i = 0; i < n; ++i) sum2_mul_add(s, c, h[i], l[i], t[i]);
    out[0] = s; out[1] = c;
    s = c = 0.f;
    for (int i = 0; i < n; ++i) sum2_add(s, c, h[i]);
    out[2] = s; out[3] = c;
}
extern "C" void roots(int n, const float *h, const float *l, float *out)
{
    for (int i = 0; i < n; ++i) out[i] = sum2_sqrt(h[i], l[i]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("sum2")
    (d / "s.cpp").write_text(CODE)
    so = str(d / "s.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}", "-o", so,
                    str(d / "s.cpp")], check=True)
    return C.CDLL(so)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("n", [1, 2, 32, 64, 65, 1120])
@pytest.mark.parametrize("kind", ["positive", "signed", "spread"])
def test_sums_against_fp64(lib, n, kind):
    rng = np.random.default_rng(n)
    v = rng.uniform(0.5, 1.5, n) if kind == "positive" else rng.normal(size=n)
    if kind == "spread":
        v *= 10.0 ** rng.uniform(-8, 3, n)
    h = v.astype(np.float32)
    l = (v - h.astype(np.float64)).astype(np.float32)
    t = np.cos(rng.uniform(0, 6.3, n)).astype(np.float32)
    out = np.zeros(4, np.float32)
    lib.sums(n, _p(h), _p(l), _p(t), _p(out))
    o, t64 = out.astype(np.float64), t.astype(np.float64)
    v2 = h.astype(np.float64) + l
    bound = n * n * 2.0 ** -48
    assert abs(o[0] + o[1] - np.sum(v2 * t64)) <= bound * np.sum(np.abs(v2 * t64))
    assert abs(o[2] + o[3] - np.sum(h.astype(np.float64))) <= bound * np.sum(np.abs(h.astype(np.float64)))


def test_root_rounds_once(lib):
    rng = np.random.default_rng(1)
    v = np.concatenate([1.0 - rng.uniform(1e-6, 1 - 1e-9, 4000) ** 2, rng.uniform(2e-9, 1.0, 4000)])
    h = v.astype(np.float32)
    l = (v - h.astype(np.float64)).astype(np.float32)
    out = np.zeros(v.size, np.float32)
    lib.roots(v.size, _p(h), _p(l), _p(out))
    r = np.sqrt(v)
    ulp = np.spacing(r.astype(np.float32)).astype(np.float64)
    assert np.all(np.abs(out.astype(np.float64) - r) <= 0.5 * ulp * (1.0 + 2.0 ** -20) + 1e-16)
