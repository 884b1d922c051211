"""A kgb_set_scene that the device has no room for (here: a direction count beyond any memory) leaves an engine without
sensors, whose traces are refused, and costs the next call nothing: the same sensors set again are traced as by an engine
that never failed."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NO_ROOM = 1 << 36   # directions: 824 GB


@pytest.fixture
def refused(engine_lib, kgb, pkg):
    """An engine that has traced 2500 sensors and was then refused all the city's sensors."""
    s = pkg.workloads.random_city(7, n_boxes=30, extent=40.0, q=1.5)
    D = pkg.workloads.hemisphere_dirs(145, 200, 5)
    e = kgb.Engine(engine_lib)
    try:
        e.build(s["v"], s["tri"])
        e.set_scene(s["P"][:2500], s["N"][:2500], D)
        e.trace(0, 2500, engine_lib.ray_flags(False, False))
        P, N = np.ascontiguousarray(s["P"], np.float32), np.ascontiguousarray(s["N"], np.float32)
        ptr = [x.ctypes.data_as(ctypes.c_void_p) for x in (P, N, D)]
        assert len(P) > 2500 and not e.d.kgb_set_scene(e.h, ptr[0], ptr[1], len(P), ptr[2], NO_ROOM)
        yield e, s, D
    finally:
        e.close()


def test_next_call_is_unharmed(refused, engine_lib, kgb):
    e, s, D = refused
    nc, flags = len(s["P"]), engine_lib.ray_flags(False, False)
    o = kgb.Engine(engine_lib)
    try:
        o.build(s["v"], s["tri"])
        o.set_scene(s["P"], s["N"], D)
        o.trace(0, nc, flags)
        for _ in range(2):   # the order made, then kept
            e.set_scene(s["P"], s["N"], D)
            e.trace(0, nc, flags)
            assert np.array_equal(e.download_bits(nc), o.download_bits(nc))
    finally:
        o.close()


def test_nothing_to_trace(refused, engine_lib, kgb):
    e, s, D = refused
    for call in (lambda: e.trace(0, 1, engine_lib.ray_flags(False, False)), lambda: e.trace(0, len(s["P"]), engine_lib.ray_flags(False, True)),
                 lambda: e.bounce(0, 1, 1, N=1, M=1, mf=1)):
        with pytest.raises(kgb.KgbError, match="range exceeds the scene"):
            call()
