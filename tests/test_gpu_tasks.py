"""The visibility kernels give the oracle's results whatever share of the directions a task takes (the launch chooses it
from the number of sensors and directions): a block per word, tasks of 8, 16 and 32 directions, ragged counts."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("nc,n_dir", [(1, 1), (33, 15), (16, 700), (2000, 31), (2001, 97), (6000, 301), (6251, 1213), (4099, 4133)])
def test_bits_bytes_views(engine_lib, oracle, kgb, pkg, nc, n_dir):
    s = pkg.workloads.random_city(3, porous=True, glass=True)
    slots = [(0.2, 0, 0, 0), (0.1, 0.4, 0, 0), (0.0, 0.64, kgb.tn_from_Tn(0.64), kgb.SLOT_GLASS), (0.2, 0, 0, 0)]
    D = pkg.workloads.hemisphere_dirs(n_dir, 1, nc)[np.random.default_rng(nc).permutation(2 * n_dir + 1)[:n_dir]]
    check = np.unique(np.concatenate([np.arange(min(nc, 40)), np.arange(max(0, nc - 40), nc)]))   # the oracle traces these
    e, o = kgb.Engine(engine_lib), kgb.Engine(oracle)
    try:
        for x, pick in ((e, np.arange(nc)), (o, check)):
            x.build(s["v"], s["tri"], s["slot"], slots, per_slot=True)
            x.set_slots(slots)
            x.set_scene(s["P"][pick], s["N"][pick], D)
        for flags in (5, 4):
            e.trace(0, nc, flags)
            o.trace(0, len(check), flags)
            a, b = (e.download_bits_rows(nc), o.download_bits_rows(len(check))) if flags == 5 else (e.download_bytes_rows(nc), o.download_bytes_rows(len(check)))
            assert np.array_equal(a[check], b)
        nAz, nEl, dAz, rowSin, _ = pkg.workloads.views_grid(120.0, 120.0 / max(1, int(n_dir ** 0.5)))
        for x, n in ((e, nc), (o, len(check))):
            x.view(0, n, 1, nAz, nEl, -60.0, dAz, rowSin, jitter=False)
        (ca, da), (cb, db) = e.download_view(nc), o.download_view(len(check))
        assert np.array_equal(ca[check], cb) and np.array_equal(da[check].view(np.uint32), db.view(np.uint32))
    finally:
        e.close()
        o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nc,n_dir", [(6000, 301), (6251, 1217), (6251, 4121), (6251, 19075)])
def test_bits_past_the_directions(engine_lib, oracle, kgb, pkg, nc, n_dir):
    """The last word's bits past the last direction are zero where tasks of 8 or 16 directions end before it, whatever the
    buffer held (a byte trace, before)."""
    s = pkg.workloads.random_city(3)
    D = pkg.workloads.hemisphere_dirs(n_dir, 1, nc)[:n_dir]
    check = np.concatenate([np.arange(16), np.arange(nc - 16, nc)])   # the oracle traces these
    e, o = kgb.Engine(engine_lib), kgb.Engine(oracle)
    try:
        for x, pick in ((e, np.arange(nc)), (o, check)):
            x.build(s["v"], s["tri"])
            x.set_scene(s["P"][pick], s["N"][pick], D)
        e.trace(0, nc, 4)
        e.trace(0, nc, 5)
        o.trace(0, len(check), 5)
        bits = e.download_bits(nc)
        assert np.array_equal(bits[:, check], o.download_bits(len(check)))
        if n_dir % 32:
            assert not np.any(bits[-1] >> np.uint32(n_dir % 32))
    finally:
        e.close()
        o.close()
