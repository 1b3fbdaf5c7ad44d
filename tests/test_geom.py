"""make_geom (csrc/common.cuh) sets every field of Geom: compiled for the host with
automatic variables filled with two different patterns, it must give the same bytes."""
import os
import shutil
import subprocess

import pytest

import ocrt_gb300

PKG = os.path.dirname(ocrt_gb300.__file__)
CUDA = "/usr/local/cuda/include"
CODE = """
#include <cuda_runtime.h>
#include "common.cuh"
#include <cstdio>
int main()
{
    for (int N = 2; N <= 64; N += 3)
        for (int E = 1; E <= 4; E += 3) {
            Geom g = make_geom(N, E);
            const int *w = (const int *)&g;
            for (size_t i = 0; i < sizeof(Geom) / 4; ++i) printf("%d ", w[i]);
            printf("\\n");
        }
}
"""


def test_every_field_is_set(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    (tmp_path / "g.cpp").write_text(CODE)
    out = []
    for init in ("zero", "pattern"):
        exe = str(tmp_path / init)
        r = subprocess.run([cxx, "-std=c++17", "-O0", "-w", f"-ftrivial-auto-var-init={init}", f"-I{PKG}/csrc",
                            f"-I{os.path.dirname(PKG)}/include", f"-I{CUDA}", "-o", exe, str(tmp_path / "g.cpp")],
                           capture_output=True, text=True)
        if "unrecognized" in r.stderr:
            pytest.skip("compiler without -ftrivial-auto-var-init")
        assert r.returncode == 0, r.stderr
        out.append(subprocess.run([exe], capture_output=True, text=True, check=True).stdout)
    assert out[0] == out[1]
