"""Tiered canvases with fewer pixel slots than blocks on outlines: the query runs
again with the exact number, and nothing learnt from the short run is kept.
Small polygons (no block is covered whole), disjoint and overlapping, so that
every overlapping pixel lies in a block the short run drops."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj

pytestmark = pytest.mark.gpu

BOX = 8000.0


def _set(overlap):
    rng = np.random.default_rng(8)
    polys = []
    for i in range(60):
        c = np.array([400.0 + 800.0 * (i % 10), 600.0 + 1200.0 * (i // 10)])
        ang = np.sort(rng.uniform(0, 2 * np.pi, 12))
        polys.append(c + rng.uniform(3.0, 14.0, (12, 1)) * np.c_[np.cos(ang), np.sin(ang)])
        if overlap:
            polys.append(polys[-1] + 2.5)
    polys += [np.array([[0.0, 0.0], [5.0, 0.0], [5.0, 5.0]]), np.array([[BOX, BOX], [BOX - 5, BOX], [BOX, BOX - 5]])]
    pidx = np.r_[0, np.cumsum([len(p) for p in polys])].astype(np.int32)
    verts = np.concatenate(polys).astype(np.float32)
    rng = np.random.default_rng(9)
    xy = np.r_[verts[rng.integers(0, len(verts), 50_000)] + rng.normal(0, 6, (50_000, 2)),
               rng.uniform(0, BOX, (10_001, 2))].astype(np.float32)
    return verts, pidx, xy


@pytest.mark.parametrize("slots", [0, 1, 40])
@pytest.mark.parametrize("overlap", [False, True])
def test_short_of_slots(built, slots, overlap):
    verts, pidx, xy = _set(overlap)
    want = oracle.raster_join(xy, verts, pidx, 1.0, max_res=1500, bounds=True)
    assert want[0].sum() > 5000 and want[2].any()
    h = rj.GLHandler()
    try:
        dh = rj.DataHandler()
        dh.add_column(1, rj.Location, xy)
        dh.setPolygons(verts, pidx)
        h.setDataHandler(dh)
        h.setCellSize(1.0)
        h.max_fbo_size = 1500
        h.flags = rj.FLAG_TIERED_CANVAS
        h.setTuning(rj.TUNE_TIER_SLOTS, slots)
        assert h.getTuning(rj.TUNE_TIER_SLOTS) == slots
        for fn in (rj.RasterJoinFn, rj.RasterJoinFn, rj.RasterJoinBoundFn):
            got = h.execute(fn)
            np.testing.assert_array_equal(got.count, want[0])
        np.testing.assert_array_equal(got.bounds, want[2])
        h.setTuning(rj.TUNE_TIER_SLOTS, -1)
        np.testing.assert_array_equal(h.execute(rj.RasterJoinFn).count, want[0])
        with pytest.raises(rj.RJError):
            h.setTuning(rj.TUNE_TIER_SLOTS, -2)
    finally:
        h.close()


@pytest.mark.parametrize("slots", [0, 1])
@pytest.mark.parametrize("overlap", [False, True])
def test_batch_short_of_slots(built, slots, overlap):
    """Batched queries run again alone, error bounds too (whose outline pass
    reads blocks that have no slot)."""
    verts, pidx, xy = _set(overlap)
    want = oracle.raster_join(xy, verts, pidx, 1.0, max_res=1500, bounds=True)
    h = rj.GLHandler()
    try:
        dh = rj.DataHandler()
        dh.add_column(1, rj.Location, xy)
        dh.setPolygons(verts, pidx)
        h.setDataHandler(dh)
        h.setCellSize(1.0)
        h.max_fbo_size = 1500
        h.flags = rj.FLAG_TIERED_CANVAS
        h.setTuning(rj.TUNE_TIER_SLOTS, slots)
        fns = [rj.RasterJoinBoundFn, rj.RasterJoinFn, rj.RasterJoinBoundFn, rj.RasterJoinFn]
        h.upload()
        got, status, _ = h.execute_batch([h.make_query(fn) for fn in fns], [None] * len(fns))
        assert not np.any(status)
        for fn, g in zip(fns, got):
            np.testing.assert_array_equal(g.count, want[0])
            if fn == rj.RasterJoinBoundFn:
                np.testing.assert_array_equal(g.bounds, want[2])
    finally:
        h.close()
