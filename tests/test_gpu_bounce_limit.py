"""A bounce whose first launch passes the time limit (lowered to a fifth of the time the whole call's kernels take) is made
of smaller launches instead, and gives the same rows, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1024, 1021])
def test_smaller_launches(engine_lib, kgb, pkg, M):
    s = pkg.workloads.random_city(44, n_boxes=300)
    nc = 4000
    assert len(s["P"]) >= nc
    e = kgb.Engine(engine_lib)
    try:
        e.build(s["v"], s["tri"], np.zeros(len(s["tri"]), np.uint32), [(0.7, 0, 0, 0)], per_slot=True)
        e.set_scene(s["P"][:nc], s["N"][:nc], np.array([[0, 0, 1]], np.float32))
        run = lambda: e.bounce(0, nc, engine_lib.bounce_flags(False), N=4, M=M, mf=1)
        run()
        rows = e.download_dc(nc)
        before = e.stats()
        run()
        now = e.stats()
        assert now["bounceLaunches"] - before["bounceLaunches"] == 1   # what the limit is a fifth of
        e.set_limits(0, bounce_limit_ns=int((now["bounceMs"] - before["bounceMs"]) * 1e6 / 5))
        run()
        assert e.stats()["bounceLaunches"] - now["bounceLaunches"] > 1
        assert np.array_equal(e.download_dc(nc).view(np.uint32), rows.view(np.uint32))
    finally:
        e.close()
