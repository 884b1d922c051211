"""The integer sums of the reduces (ordered_sum.cuh) give the bits of a chain of double fmas, after every term (CPU), and
the reduces that use them the oracle's doubles (GPU)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import REPO

SO = os.path.join(REPO, "tests", "_build", "ordered_sum_check.so")


@pytest.fixture(scope="module")
def checker():
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", SO, os.path.join(REPO, "tests", "ordered_sum_check.cpp")])
    lib = ctypes.CDLL(SO)
    lib.ordered_sum_check.argtypes = [ctypes.c_int, ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
    return lib


@pytest.mark.parametrize("kind", range(7))
def test_terms(checker, kind):
    out = (ctypes.c_uint64 * 2)()
    checker.ordered_sum_check(kind, 1, 200 if kind == 0 else 10000, out)
    assert out[0] > 100000 and out[1] == 0


def weights(n, kind, rng):
    w = rng.uniform(0, 1, n).astype(np.float32)
    if kind == "powers":
        w = np.ldexp(np.float32(1), rng.integers(-40, 40, n)).astype(np.float32)
    elif kind == "range":
        w = (w * np.ldexp(np.float32(1), rng.integers(-100, 100, n))).astype(np.float32)
    elif kind == "zeros":
        w[rng.random(n) < 0.7] = 0
    elif kind == "whole":
        w = rng.integers(0, 9, n).astype(np.float32)
    elif kind == "negative":
        w -= np.float32(0.5)
    elif kind == "subnormal":
        w[::3] = np.float32(1e-41)
    elif kind == "huge":
        w *= np.float32(3e38)
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("n_dir", [1, 255, 256, 259, 700])
@pytest.mark.parametrize("nc", [1, 5, 130, 2000])
def test_reduces(engine_lib, oracle, kgb, pkg, n_dir, nc):
    s = pkg.workloads.random_city(5, porous=True, glass=True)
    slots = [(0.2, 0, 0, 0), (0.1, 0.4, 0, 0), (0.0, 0.64, kgb.tn_from_Tn(0.64), kgb.SLOT_GLASS), (0.2, 0, 0, 0)]
    rng = np.random.default_rng(n_dir * 7 + nc)
    D = pkg.workloads.hemisphere_dirs(n_dir, 1, 3)[rng.permutation(2 * n_dir + 1)[:n_dir]]
    pick = rng.permutation(len(s["P"]))[:nc]
    N = s["N"][pick].copy()
    if nc > 1:
        N[1] = (0.0, 0.0, 3e-42)   # its cosines are not normal floats
    e, o = kgb.Engine(engine_lib), kgb.Engine(oracle)
    try:
        for x in (e, o):
            x.build(s["v"], s["tri"], s["slot"], slots, per_slot=True)
            x.set_slots(slots)
            x.set_scene(s["P"][pick], N, D)
        for flags in (5, 4):
            for x in (e, o):
                x.trace(0, nc, flags)
            for kind in ("uniform", "powers", "range", "zeros", "whole", "negative", "subnormal", "huge"):
                W = weights(n_dir, kind, rng)
                for cos in (True, False):
                    a, b = e.reduce(nc, W, cos), o.reduce(nc, W, cos)
                    assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), (flags, kind, cos)
        if n_dir == 259:
            for x in (e, o):
                x.set_scene(s["P"][pick], s["N"][pick], D)
                x.bounce(0, nc, 1, N=1, M=16, mf=1)
            for kind in ("uniform", "powers", "zeros", "negative", "subnormal"):
                W = weights(146, kind, rng)
                assert np.array_equal(e.reduce_dc(nc, W).view(np.uint64), o.reduce_dc(nc, W).view(np.uint64)), kind
    finally:
        e.close()
        o.close()
