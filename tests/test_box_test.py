"""The traversal's box test is conservative (CPU): the device code of rt.cuh, compiled for the CPU, finds for every ray
exactly the hits that a loop over all triangles finds, and the same closest one (tests/box_test_check.cpp)."""
import ctypes
import os
import subprocess

import pytest

from conftest import REPO

SO = os.path.join(REPO, "tests", "_build", "box_test_check.so")


@pytest.fixture(scope="module")
def checker():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    src = [os.path.join(REPO, "tests", "box_test_check.cpp"), os.path.join(REPO, "kit-sim_daylight_gb300", "csrc", "bvh_build.cpp")]
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I" + os.path.join(REPO, "include"),
                           "-I/usr/local/cuda/include", "-o", SO] + src)
    lib = ctypes.CDLL(SO)
    lib.box_test_check.argtypes = [ctypes.c_uint64, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
    return lib


@pytest.mark.parametrize("kind", range(8))   # four scales (largest coordinate 1, 40, 500, 20000), walls along the axes or turned
def test_walk_finds_every_hit(checker, kind):
    out = (ctypes.c_uint64 * 4)()
    for seed in range(3):
        checker.box_test_check(seed, kind, 4000, out)
    assert out[0] > 10000 and out[1] > out[0] // 2
    assert out[2] == 0 and out[3] == 0
