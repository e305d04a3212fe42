"""The lanes that a shuffle of the edge kernels names take the same branch (CPU: the kernels' own index
rules over the lists of real parts)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cuteflow_gb300 import _abi, cases, domains

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("lanes") / "liblanes.so")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-deprecated-declarations",
                    "-I", cuda_inc, "-I", os.path.join(ROOT, "include"), "-o", out,
                    os.path.join(HERE, "lanes_harness.cpp"),
                    os.path.join(ROOT, "cuteflow_gb300", "csrc", "cf_mesh.cpp")], check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("nparts", [2, 3])
@pytest.mark.parametrize("iflux", [1, 3])
def test_a_warp_of_a_parts_list_has_one_arithmetic_type(lib, iflux, nparts):
    parts = domains.partition(cases.flooding(40, 20, seed=4, iflux=iflux), nparts)
    by_number = 0
    for rank, p in enumerate(parts):
        ma, prm = _abi.MeshArrays(p.case), _abi.make_params({**p.case.params, **p.params})
        cls = np.ascontiguousarray(domains.part_plan(parts, rank)[0], np.int32)
        for mask in range(32):
            n = [C.c_int32() for _ in range(3)]
            assert lib.harness_list_warps(C.byref(ma.mesh), C.byref(prm), cls.ctypes.data_as(C.POINTER(C.c_int32)),
                                          mask, *[C.byref(x) for x in n]) == 0
            assert n[0].value > 0 and n[1].value == 0
            by_number += n[2].value
    assert by_number > 0   # the lists do hold warps whose edges' numbers differ in the mask's bit


def test_a_recording_forward_takes_the_shape_that_was_set(lib):
    out = (C.c_int32 * 2)()
    for eb in (64, 128, 256):
        for ept in (1, 2):
            lib.harness_recording_shape(eb, ept, 1, out)
            assert tuple(out) == (eb, ept)
            lib.harness_recording_shape(eb, ept, 0, out)
            assert tuple(out) == (256, 1)


def test_the_lines_of_the_dispatch_follow_the_number_of_sms(lib):
    lib.harness_edge_block.argtypes = [C.c_longlong, C.c_int32]
    for sms in (152, 76, 132):
        assert lib.harness_edge_block(512 * sms, sms) == 64 and lib.harness_edge_block(512 * sms + 128, sms) == 256
        assert lib.harness_two_lanes(sms, sms) == 1 and lib.harness_two_lanes(sms + 1, sms) == 0
        assert [lib.harness_adj_blocks(n, sms) for n in (3 * sms, 3 * sms + 1, 4 * sms, 4 * sms + 1)] == [3, 4, 4, 3]
    assert lib.harness_edge_block(1 << 30, 152) == 256   # no overflow at the largest context
