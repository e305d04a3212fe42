"""The edge that the reverse sweep differentiates as a whole is the one that the step evaluates from its two
sides, standing waves included: every branch of the one is the other's (CPU build of the same code)."""
import ctypes as C
import os
import platform
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("forms") / "libforms.so")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    extra = ["-mfma"] if platform.machine() == "x86_64" else []
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off"] + extra + [
                    "-Wno-deprecated-declarations", "-I", cuda_inc, "-I", os.path.join(ROOT, "include"), "-o", out,
                    os.path.join(HERE, "forms_harness.cpp")], check=True)
    L = C.CDLL(out)
    L.harness_forms.argtypes = [C.c_int, C.c_longlong, C.c_ulonglong, C.POINTER(C.c_longlong)]
    L.harness_forms.restype = C.c_longlong
    return L


@pytest.mark.parametrize("iflux", [1, 2, 3])
def test_the_differentiated_edge_is_the_steps(lib, iflux):
    standing = C.c_longlong()
    assert lib.harness_forms(iflux, 200_000, 5, C.byref(standing)) == 0
    assert standing.value > 10_000   # 15 % of the edges
