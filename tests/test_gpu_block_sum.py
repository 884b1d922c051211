"""Reduces of few sensors over many directions (a block a sensor) give the oracle's doubles, at the edges of the sizes that
take this form and for weights whose sums leave their binade often, meet halfway terms in every word, or are not sums of
normal products."""
import numpy as np
import pytest


def weights(n, kind, rng):
    w = rng.uniform(0, 1, n).astype(np.float32)
    if kind == "powers":
        w = np.ldexp(np.float32(1), rng.integers(-40, 40, n)).astype(np.float32)
    elif kind == "rising":
        w = np.ldexp(w, np.arange(n) // 50).astype(np.float32)
    elif kind == "zeros":
        w[rng.random(n) < 0.9] = 0
    elif kind == "halfway":   # sums of 2^30 to 2^37, whose last bits are 2^-22 to 2^-15, and odd multiples of half of these
        w = np.ldexp((2 * rng.integers(0, 1000, n) + 1).astype(np.float32), -rng.integers(16, 24, n)).astype(np.float32)
        w[rng.random(n) < 0.02] = 2.0 ** 30
    elif kind == "late":      # nothing, or little, before the last terms
        w[: n - 40] *= np.float32(1e-30)
        w[: n // 2] = 0
    elif kind == "subnormal":
        w[::3] = np.float32(1e-41)
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("nc,n_dir", [(1, 2047), (1, 2048), (5, 2303), (16, 4133), (450, 2049), (451, 2049)])
def test_reduces(engine_lib, oracle, kgb, pkg, nc, n_dir):
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
            for kind in ("uniform", "powers", "rising", "zeros", "halfway", "late", "subnormal"):
                W = weights(n_dir, kind, rng)
                for cos in (True, False):
                    a, b = e.reduce(nc, W, cos), o.reduce(nc, W, cos)
                    assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), (flags, kind, cos)
        for x in (e, o):
            x.bounce(0, nc, 1, N=1, M=64, mf=4)
        for kind in ("uniform", "powers", "halfway", "late", "subnormal"):
            W = weights(2306, kind, rng)
            assert np.array_equal(e.reduce_dc(nc, W).view(np.uint64), o.reduce_dc(nc, W).view(np.uint64)), kind
    finally:
        e.close()
        o.close()
