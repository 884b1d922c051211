"""A warp's frontier, built on the CPU by the device code (tests/frontier_check.cpp): in a sound tree its subtrees hold every
triangle exactly once; in a damaged one the build ends all the same."""
import ctypes
import os
import subprocess

import pytest

from conftest import REPO

SO = os.path.join(REPO, "tests", "_build", "frontier_check.so")


@pytest.fixture(scope="module")
def checker():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    src = [os.path.join(REPO, "tests", "frontier_check.cpp"), os.path.join(REPO, "kit-sim_daylight_gb300", "csrc", "bvh_build.cpp")]
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-I" + os.path.join(REPO, "include"),
                           "-I/usr/local/cuda/include", "-o", SO] + src)
    lib = ctypes.CDLL(SO)
    lib.frontier_check.argtypes = [ctypes.c_uint64, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_uint32)]
    return lib


@pytest.mark.parametrize("spread", [0, 1, 2])   # origins a few metres apart, all over the scene, together with some not finite
@pytest.mark.parametrize("seed", [1, 2, 5])     # 5: one triangle
def test_holds_every_triangle(checker, seed, spread):
    n = ctypes.c_uint32(0)
    assert checker.frontier_check(seed, 0, spread, n) == 0
    assert n.value >= (1 if seed == 5 else 8)


@pytest.mark.parametrize("damage", [1, 2])
@pytest.mark.parametrize("spread", [0, 1])
def test_ends_in_damaged_trees(checker, damage, spread):
    n = ctypes.c_uint32(0)
    assert checker.frontier_check(1, damage, spread, n) == 0
