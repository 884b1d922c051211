"""A sensor whose position or normal is not finite changes no other sensor's result: traces large enough to walk from
frontiers, which a warp's sensors share, and served requests give the other sensors what they have without it, and every
sensor what small traces, which walk from the root, give it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spoil(P, N, at):
    """Positions and normals that are not finite, of every kind, at the sensors `at`."""
    P, N = P.copy(), N.copy()
    bad = np.array([np.nan, -np.nan, np.inf, -np.inf], np.float32)
    for k, i in enumerate(at):
        if k % 9 == 8:
            P[i] = 0.001   # a normal that is not finite moves only an origin near zero by its product
            N[i, k % 3] = bad[k % 4]
        else:
            P[i, k % 3] = bad[k % 4]
    return P, N


@pytest.mark.parametrize("scene", ["city", "block"])
def test_traces(engine_lib, oracle, kgb, pkg, scene):
    n_dir, n = 2400, 6251
    rng = np.random.default_rng(1)
    if scene == "block":
        s = pkg.workloads.urban_block(seed=3, n=6, target_sensors=n + 500, glass_share=0.2)
        P, N = s["P"][:n], s["N"][:n]
    else:
        s = pkg.workloads.random_city(3, porous=True, glass=True)
        pick = np.sort(rng.integers(0, len(s["P"]), n))
        P, N = s["P"][pick], s["N"][pick]
    slots = [(0.2, 0, 0, 0), (0.1, 0.4, 0, 0), (0.0, 0.64, kgb.tn_from_Tn(0.64), kgb.SLOT_GLASS), (0.2, 0, 0, 0)]
    D = pkg.workloads.hemisphere_dirs(n_dir // 2, 0, 3)
    bad = np.sort(rng.choice(n, n // 40, replace=False))
    good = np.setdiff1d(np.arange(n), bad)
    check = rng.choice(good, 160, replace=False)
    P2, N2 = spoil(P, N, bad)
    e, o = kgb.Engine(engine_lib), kgb.Engine(oracle)
    try:
        for x, p, m in ((e, P2, N2), (o, P[check], N[check])):
            x.build(s["v"], s["tri"], np.minimum(s["slot"], 3), slots, per_slot=True)
            x.set_slots(slots)
            x.set_scene(p, m, D)
        for flags in (5, 4):
            down = (lambda x, k: x.download_bits(k)) if flags == 5 else (lambda x, k: x.download_bytes(k))
            e.trace(0, n, flags)
            whole = down(e, n)
            o.trace(0, len(check), flags)
            assert np.array_equal(whole[:, check], down(o, len(check))), flags
            for i0 in range(0, n, 1000):   # too few rays for frontiers
                m = min(1000, n - i0)
                e.trace(i0, m, flags)
                assert np.array_equal(down(e, m), whole[:, i0:i0 + m]), (flags, i0)
    finally:
        e.close()
        o.close()


@pytest.mark.parametrize("n_dir", [40, 300])
def test_served_request(engine_lib, kgb, pkg, n_dir):
    s = pkg.workloads.random_city(4, n_boxes=60)
    rng = np.random.default_rng(n_dir)
    n = 1500
    P, N = s["P"][:n], s["N"][:n]
    D = pkg.workloads.hemisphere_dirs(n_dir // 2, 0, 5)
    W = rng.uniform(0.1, 2.0, (2, len(D))).astype(np.float32)
    bad = np.sort(rng.choice(n, n // 30, replace=False))
    P2, N2 = spoil(P, N, bad)
    srv = kgb.Server(engine_lib, 1e9)
    try:
        sid = srv.add_scene(s["v"], s["tri"])
        got = srv.wait(srv.submit(sid, P2, N2, D, W, [True, False]))
        want = srv.wait(srv.submit(sid, P, N, D, W, [True, False]))
    finally:
        srv.close()
    good = np.setdiff1d(np.arange(n), bad)
    assert np.array_equal(got[:, good], want[:, good])
    e = kgb.Engine(engine_lib)
    try:
        e.build(s["v"], s["tri"])
        e.set_scene(P, N, D)
        e.trace(0, n, engine_lib.ray_flags(False, False))
        for q, cos in enumerate((True, False)):
            assert np.array_equal(want[q], e.reduce(n, W[q], cos))
    finally:
        e.close()
