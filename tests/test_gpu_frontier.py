"""Traces large enough to walk from frontiers (at least 96 directions and 2^23 rays a launch) give the oracle's bits and
bytes on sampled sensors: dense and scattered sensors, sensors far outside the scene, a scene of few triangles, directions
along the axes."""
import numpy as np
import pytest


def directions(pkg, n):
    D = pkg.workloads.hemisphere_dirs(n // 2, n - 2 * (n // 2), 3)
    D[:6] = [[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]]
    return np.ascontiguousarray(D[:n])


@pytest.mark.gpu
@pytest.mark.parametrize("scene,n_dir", [("city", 1400), ("city", 96), ("block", 1401), ("box", 1402), ("far", 1400)])
def test_bits_and_bytes(engine_lib, oracle, kgb, pkg, scene, n_dir):
    rng = np.random.default_rng(n_dir)
    n = max(6251, -(-(1 << 23) // n_dir) + 5)
    if scene == "block":
        s = pkg.workloads.urban_block(seed=3, n=6, target_sensors=n + 500, glass_share=0.2)
        P, N = s["P"][:n], s["N"][:n]
    else:
        s = pkg.workloads.box_scene() if scene == "box" else pkg.workloads.random_city(3, porous=True, glass=True)
        pick = rng.integers(0, len(s["P"]), n)
        P, N = s["P"][pick].copy(), s["N"][pick].copy()
        if scene == "far":
            P[::2] += rng.normal(size=(len(P[::2]), 3)).astype(np.float32) * 3000
            N[::2] = -P[::2] / np.linalg.norm(P[::2], axis=1, keepdims=True)
        if scene == "box":
            P += rng.uniform(-0.4, 0.4, P.shape).astype(np.float32)
    n = len(P)
    slots = [(0.2, 0, 0, 0), (0.1, 0.4, 0, 0), (0.0, 0.64, kgb.tn_from_Tn(0.64), kgb.SLOT_GLASS), (0.2, 0, 0, 0)]
    slot = np.minimum(s["slot"], 3)
    D = directions(pkg, n_dir)
    check = np.sort(rng.choice(n, 160, replace=False))
    e, o = kgb.Engine(engine_lib), kgb.Engine(oracle)
    try:
        for x, at in ((e, np.arange(n)), (o, check)):
            x.build(s["v"], s["tri"], slot, slots, per_slot=True)
            x.set_slots(slots)
            x.set_scene(P[at], N[at], D)
        for flags in (5, 21, 4):
            e.trace(0, n, flags)
            o.trace(0, len(check), flags)
            a, b = (e.download_bits(n), o.download_bits(len(check))) if flags != 4 else (e.download_bytes(n), o.download_bytes(len(check)))
            assert np.array_equal(a[:, check], b), flags
    finally:
        e.close()
        o.close()
