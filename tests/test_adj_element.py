"""The transposed element stage of the reverse sweep against the element stage differentiated by dual
numbers, for every friction option (CPU build of the same code)."""
import ctypes as C
import os
import platform
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("element") / "libelement.so")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    extra = ["-mfma"] if platform.machine() == "x86_64" else []
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off"] + extra + [
                    "-Wno-deprecated-declarations", "-I", cuda_inc, "-I", os.path.join(ROOT, "include"), "-o", out,
                    os.path.join(HERE, "element_harness.cpp")], check=True)
    L = C.CDLL(out)
    L.harness_adj_element.argtypes = [C.c_longlong, C.c_ulonglong, C.c_int, C.c_int]
    L.harness_adj_element.restype = C.c_double
    return L


@pytest.mark.parametrize("friction,fricimplic", [(0, 0), (1, 0), (1, 1), (1, 2)])
def test_transposed_element_is_the_dual_derivative(lib, friction, fricimplic):
    # ~30 operations on either side, each within 2^-53 of terms no larger than the largest contribution
    # but for cancellations of a factor ~100
    assert lib.harness_adj_element(200_000, 3, friction, fricimplic) < 1e-12


def test_reverse_edge_with_a_nearly_dry_side_is_the_dual_derivative(lib):
    lib.harness_adj_nearly_dry.argtypes = [C.c_longlong, C.c_ulonglong]
    lib.harness_adj_nearly_dry.restype = C.c_double
    assert lib.harness_adj_nearly_dry(200_000, 9) < 1e-12


def test_element_by_two_lanes_is_the_element(lib):
    lib.harness_element_pair.argtypes = [C.c_longlong, C.c_ulonglong]
    lib.harness_element_pair.restype = C.c_longlong
    assert lib.harness_element_pair(600_000, 17) == 0
