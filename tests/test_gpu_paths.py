"""Reflected light gives the oracle's rows, bit for bit, whatever the numbers of paths: none or few to take from the queue,
a queue far longer than the GPU's lanes, paths of many segments (glass, porous and thin panes), ragged sample counts."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nc,M,N", [(1, 1, 1), (1, 1000, 0), (33, 7, 5), (257, 129, 2), (4001, 9, 1), (4001, 16, 1), (3000, 65, 3)])
def test_rows(engine_lib, oracle, kgb, pkg, nc, M, N):
    s = pkg.workloads.random_city(5, porous=True, glass=True, thin=True)
    slots = [(0.2, 0, 0, 0), (0.3, 0.5, 0, 0), (0.0, 0.64, kgb.tn_from_Tn(0.64), kgb.SLOT_GLASS), (0.25, 0, 0, 0), (0.2, 0, 0, 0),
             (0.2, 0, 0, 0), (0.2, 0, 0, 0), (0.1, 0.6, 0, kgb.SLOT_THIN)]
    rows = []
    for lib in (engine_lib, oracle):
        e = kgb.Engine(lib)
        try:
            e.build(s["v"], s["tri"], s["slot"], slots, per_slot=True)
            e.set_slots(slots)
            e.set_scene(s["P"][:nc], s["N"][:nc], np.array([[0, 0, 1]], np.float32))
            e.bounce(0, nc, lib.bounce_flags(False), N=N, M=M, mf=2, north=20.0)
            rows.append(e.download_dc(nc))
        finally:
            e.close()
    assert np.array_equal(rows[0].view(np.uint32), rows[1].view(np.uint32))
