"""The time series runs a chunk in bands of 128-sensor tile rows, as many as its sizes make worth while: the rows of E are
those that chunks of one tile row give (one band each), bit for bit, over counts that leave ragged last bands, tiles and
columns, for visibility as bits and as bytes."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("P,nc,T,as_bytes", [(145, 1, 1, False), (145, 129, 65, True), (600, 3001, 1999, False), (2305, 385, 8760, True),
                                             (2305, 1030, 4449, False), (2305, 4700, 2221, True), (2305, 4999, 4456, False)])
def test_bands(engine_lib, kgb, pkg, P, nc, T, as_bytes):
    s = pkg.workloads.random_city(8, n_boxes=40)
    rng = np.random.default_rng(nc)
    nSun = (T + 1) // 2   # half the columns have a sun direction, in no order
    D = pkg.workloads.hemisphere_dirs(P, nSun, 8)
    e = kgb.Engine(engine_lib)
    try:
        e.build(s["v"], s["tri"])
        e.set_scene(s["P"][:nc], s["N"][:nc], D)
        args = dict(nSky=P, row=np.arange(P), wsky=np.full(P, 2 * np.pi / P, np.float32), S=rng.gamma(2.0, 30.0, (P, T)).astype(np.float32),
                    g=rng.uniform(5, 40, T).astype(np.float32), sun0=2 * P, sunStep=rng.permutation(T)[:nSun].astype(np.int32),
                    sunVec=D[2 * P:], sunW=rng.uniform(100, 900, nSun).astype(np.float32))
        G = rng.uniform(0.1, 1.0, nc).astype(np.float32)
        flags = engine_lib.ray_flags(False, as_bytes)
        e.trace(0, nc, flags)
        whole = e.series(nc, G=G, **args)
        for i0 in range(0, nc, 128):
            m = min(128, nc - i0)
            e.trace(i0, m, engine_lib.ray_flags(False, False))   # an opaque scene: its bytes are its bits
            assert np.array_equal(e.series(m, G=G[i0:i0 + m], **args), whole[i0:i0 + m])
        assert np.abs(whole).max() > 0
    finally:
        e.close()
