"""Tiered canvases under a memory budget that holds the pixel slots the outlines
need, but not as many as their vertices could: every form joins, equal to the
results without a budget.  Small polygons of many vertices on 20,000 x 20,000
pixels: at most 20,000 blocks on outlines where the bound is 338,000 (173 MB of
labels, 346 MB of counts, beside some 50 MB that is not slots)."""
import numpy as np
import pytest

import rasterjoin as rj

pytestmark = pytest.mark.gpu

BOX = 40000.0
N = 100_001


def _rings(overlap):
    rng = np.random.default_rng(3)
    polys = []
    for i in range(100 if overlap else 200):
        c = 1000.0 + 2000.0 * np.array([i % 20, i // 20 * 2])
        ang = np.sort(rng.uniform(0, 2 * np.pi, 100))
        rad = rng.uniform(60.0, 140.0, 100)
        polys.append(c + rad[:, None] * np.c_[np.cos(ang), np.sin(ang)])
        if overlap:
            polys.append(polys[-1] + 40.0)
    polys += [np.array([[0.0, 0.0], [9.0, 0.0], [9.0, 9.0]]), np.array([[BOX, BOX], [BOX - 9, BOX], [BOX, BOX - 9]])]
    pidx = np.r_[0, np.cumsum([len(p) for p in polys])].astype(np.int32)
    rng = np.random.default_rng(4)
    near = np.concatenate(polys)[rng.integers(0, pidx[-1], N - 20_000)] + rng.normal(0, 30, (N - 20_000, 2))
    xy = np.r_[near, rng.uniform(0, BOX, (20_000, 2))].astype(np.float32)
    return np.concatenate(polys).astype(np.float32), pidx, xy


def _handler(mb, verts, pidx, xy):
    h = rj.GLHandler(gpu_mem_mb=mb)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.add_column(2, rj.Float, np.random.default_rng(6).lognormal(2.5, 0.8, N).astype(np.float32))
    dh.setPolygons(verts, pidx)
    h.setDataHandler(dh)
    h.setCellSize(2.0)
    h.flags = rj.FLAG_TIERED_CANVAS
    return h, dh


def _queries(h, dh):
    for fn, aggr in ((rj.RasterJoinFn, False), (rj.RasterJoinFn, True), (rj.RasterJoinBoundFn, False)):
        dh.setAggregation(rj.Sum if aggr else rj.Count, 2 if aggr else -1)
        yield fn, h.make_query(fn)


def _same(got, want):
    np.testing.assert_array_equal(got.count, want.count)
    np.testing.assert_array_equal(got.sum, want.sum)
    if want.bounds is not None:
        np.testing.assert_array_equal(got.bounds, want.bounds)


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("batch", [False, True])
def test_budget_between_exact_and_bound(built, overlap, batch):
    verts, pidx, xy = _rings(overlap)
    free, dh = _handler(0, verts, pidx, xy)
    tight, dt = _handler(150, verts, pidx, xy)
    try:
        want = [free.execute(fn, q) for fn, q in _queries(free, dh)]
        assert want[0].count.sum() > 10_000
        qs = list(_queries(tight, dt))
        if batch:
            tight.upload()
            got = tight.execute_batch([q for _, q in qs], [None] * len(qs))[0]
        else:
            got = [tight.execute(fn, q) for fn, q in qs]
        for g, w in zip(got, want):
            _same(g, w)
    finally:
        free.close()
        tight.close()


@pytest.mark.parametrize("overlap,mb", [(False, 124), (True, 368)])
def test_one_tile_budget_of_the_flat_map(built, overlap, mb):
    """A budget that holds a flat label map of 8000 x 8000 pixels (128 MB; with
    the counts of overlapping polygons 384), but not the blocks, which take 3 %
    more: the query and a plan of it run, equal to those without a budget."""
    rng = np.random.default_rng(5)
    polys = [np.array([[x, y], [x + w, y], [x + w, y + w], [x, y + w]]) for x in range(0, 8000, 1000) for y in range(0, 8000, 1000)
             for w in ((1000, 700) if overlap and (x + y) % 3000 == 0 else (1000,))]
    verts = np.concatenate(polys).astype(np.float32)
    pidx = 4 * np.arange(len(polys) + 1, dtype=np.int32)
    xy = rng.uniform(-10, 8010, (5001, 2)).astype(np.float32)
    got = []
    for budget in (0, mb):
        h = rj.GLHandler(gpu_mem_mb=budget)
        try:
            dh = rj.DataHandler()
            dh.add_column(1, rj.Location, xy)
            dh.setPolygons(verts, pidx)
            h.setDataHandler(dh)
            h.setCellSize(1.0)
            h.flags = rj.FLAG_FLAT_CANVAS
            got.append(h.execute(rj.RasterJoinFn))
            got.append(h.execute(rj.RasterJoinFn))
            plan = h.prepare(rj.RasterJoinFn)
            got.append(plan.execute())
            plan.close()
        finally:
            h.close()
    assert got[0].count.sum() > 4900
    for g in got[1:]:
        np.testing.assert_array_equal(g.count, got[0].count)


def test_phase_times_without_room_for_the_block_codes(built):
    """Tables that leave room for the blocks of 4000 x 4000 pixels, for these
    without the 125 KB of their codes, or for the flat label map only: the same
    counts, and the phases are timed, call after call."""
    polys = [np.array([[x, y], [x + 500, y], [x + 500, y + 500], [x, y + 500]]) for x in range(0, 4000, 500)
             for y in range(0, 4000, 500)]
    verts = np.concatenate(polys).astype(np.float32)
    pidx = 4 * np.arange(len(polys) + 1, dtype=np.int32)
    rows = range(1_030_000, 1_180_000, 12_288)   # 96 KB each
    xy = np.random.default_rng(5).uniform(1, 3999, (rows[-1], 2)).astype(np.float32)
    lean = []
    for n in rows:
        got = []
        for budget in (0, 40):
            h = rj.GLHandler(gpu_mem_mb=budget)
            try:
                dh = rj.DataHandler()
                dh.add_column(1, rj.Location, xy[:n])
                dh.setPolygons(verts, pidx)
                h.setDataHandler(dh)
                h.setCellSize(1.0)
                h.flags = rj.FLAG_FLAT_CANVAS | rj.FLAG_PHASE_TIMING
                h.setTuning(rj.TUNE_COUNT_BLOCK_SHIFT, 4)
                for _ in range(3):
                    got.append(h.execute(rj.RasterJoinFn))
                    t = h.timings()
                    assert t["poly_render_ms"] > 0 and t["pt_render_ms"] > 0
                if budget:
                    lean.append(h.getTuning(rj.TUNE_COUNT_SHAPE) >= 0)
            finally:
                h.close()
        assert got[0].count.sum() >= n
        for g in got[1:]:
            np.testing.assert_array_equal(g.count, got[0].count)
    assert lean[0] and not lean[-1]
