"""Rays that start just past a triangle's edge and leave it almost along its plane (CPU; tests/edge_ray_check.cpp): the walk
finds the hits of a loop over all triangles, and the same closest one. There the computed hit distance is off by a
rounding error of the triangle's extent over the sine of the ray against the plane, more than any box allows for in the
end; what has to hold is that no hit is lost which a box expanded by 2^-16 of the scene's largest coordinate keeps."""
import ctypes
import os
import subprocess

import pytest

from conftest import REPO

SO = os.path.join(REPO, "tests", "_build", "edge_ray_check.so")


@pytest.fixture(scope="module")
def checker():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    src = [os.path.join(REPO, "tests", "edge_ray_check.cpp"), os.path.join(REPO, "kit-sim_daylight_gb300", "csrc", "bvh_build.cpp")]
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I" + os.path.join(REPO, "include"),
                           "-I/usr/local/cuda/include", "-o", SO] + src)
    lib = ctypes.CDLL(SO)
    lib.edge_ray_check.argtypes = [ctypes.c_uint64, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
    return lib


@pytest.mark.parametrize("kind", range(8))   # four scales (largest coordinate 1, 40, 500, 20000), walls along the axes or turned
def test_walk_finds_every_hit(checker, kind):
    out = (ctypes.c_uint64 * 5)()
    for seed in range(3):
        checker.edge_ray_check(seed, kind, 40000, out)
    assert out[0] > 100000 and out[1] > out[0] // 4 and out[4] < 10
    assert out[2] == 0 and out[3] == 0
