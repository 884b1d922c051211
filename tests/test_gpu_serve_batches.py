"""Served daylight batches on both sides of the size from which a warp takes two tasks at a time (four tasks for each of the
grid's 32 warps an SM) give the sums of the single-request engine, bit for bit: batches well below it, just above and below
it by odd counts, and of two requests that meet within a warp's two tasks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_dir,tasks", [(14, -19000), (256, -8), (256, 8), (257, 9), (33, 1)])
def test_equal_alone(engine_lib, kgb, pkg, n_dir, tasks):
    import torch
    line = 4 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    words = (n_dir + 31) // 32
    n = (line + tasks) // words * 32 + (1 if tasks > 0 else 0)   # sensors of both requests together
    s = pkg.workloads.random_city(9, n_boxes=40)
    rng = np.random.default_rng(n_dir)
    pick = rng.integers(0, len(s["P"]), n)
    P, N = s["P"][pick], s["N"][pick]
    D = pkg.workloads.hemisphere_dirs(n_dir, 1, 2)[rng.permutation(2 * n_dir + 1)[:n_dir]]
    W = rng.uniform(0.1, 2.0, (1, n_dir)).astype(np.float32)
    cut = n // 3 // 32 * 32 + 5
    srv = kgb.Server(engine_lib, 8e9)
    try:
        sid = srv.add_scene(s["v"], s["tri"])
        srv.set_tuning(chunk_sensors=1 << 18, batch_rays=1 << 28, view_rays=1 << 16)
        t = [srv.submit(sid, P[a:b], N[a:b], D, W, [True]) for a, b in ((0, cut), (cut, n))]
        got = np.concatenate([srv.wait(x)[0] for x in t])
    finally:
        srv.close()
    e = kgb.Engine(engine_lib)
    try:
        e.build(s["v"], s["tri"])
        e.set_scene(P, N, D)
        e.trace(0, n, engine_lib.ray_flags(False, False))
        assert np.array_equal(got, e.reduce(n, W[0], True))
    finally:
        e.close()
