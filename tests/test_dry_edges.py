"""The slots of an edge between two dry elements, written without evaluating it, are the bits that the step's
own two-sided evaluation gives (CPU build of the same code)."""
import ctypes as C
import os
import platform
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("dry") / "libdry.so")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    extra = ["-mfma"] if platform.machine() == "x86_64" else []
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off"] + extra + [
                    "-Wno-deprecated-declarations", "-I", cuda_inc, "-I", os.path.join(ROOT, "include"), "-o", out,
                    os.path.join(HERE, "dry_harness.cpp")], check=True)
    L = C.CDLL(out)
    L.harness_dry_edges.argtypes = [C.c_longlong, C.c_ulonglong, C.c_int, C.POINTER(C.c_longlong)]
    L.harness_dry_edges.restype = C.c_longlong
    return L


@pytest.mark.parametrize("iflux", [1, 2, 3, 4])
def test_dry_slots_are_the_steps(lib, iflux):
    took = C.c_longlong()
    assert lib.harness_dry_edges(400_000, 21 + iflux, iflux, C.byref(took)) == 0
    assert took.value > 200_000
