"""Tiled canvases so far from the origin (in pixels) that fp32 moves a point by
whole pixels: neighbouring tiles disagree on where it lies by more than a pixel.
Points around the seams and the rim, every form, against the oracle."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu


def _run(handler, lo, ext, fbo, polygons):
    verts, pidx = polygons
    verts = (verts.astype(np.float64) + lo).astype(np.float32)
    bb = np.r_[verts.min(0), verts.max(0)].astype(np.float64)
    rng = np.random.default_rng(fbo)
    xy = rng.uniform(bb[:2] - 30, bb[2:] + 30, (150_001, 2))
    split = int(np.ceil(np.ceil(ext) / fbo))
    for k in range(2):
        i = slice(k * 50_000, (k + 1) * 50_000)
        xy[i, k] = bb[k] + rng.integers(0, split + 1, 50_000) * (bb[2 + k] - bb[k]) / split + rng.uniform(-14, 14, 50_000)
    xy = xy.astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setCellSize(1.0)
    handler.max_fbo_size = fbo
    want = oracle.raster_join(xy, verts, pidx, 1.0, max_res=fbo, bounds=True)
    assert want[0].sum() > 50_000
    try:
        for fn, flag in ((rj.RasterJoinFn, 0), (rj.RasterJoinFn, rj.FLAG_FORCE_CANVAS), (rj.RasterJoinBoundFn, 0)):
            handler.flags = rj.FLAG_TIERED_CANVAS | flag
            got = handler.execute(fn)
            assert handler.getTuning(rj.TUNE_COUNT_SHAPE) >= 0      # a lean pass ran
            np.testing.assert_array_equal(got.count, want[0])
        np.testing.assert_array_equal(got.bounds, want[2])
    finally:
        handler.flags = 0
        handler.max_fbo_size = 8192


@pytest.mark.parametrize("lo,ext,fbo", [((9565671.0, 9565671.0), 8850.0, 943), ((500000.0, 4100000.0), 6000.0, 1700),
                                        ((-10160196.0, 4100000.0), 8718.0, 1679), ((36316732.0, -36316732.0), 5064.0, 876)])
def test_seams(handler, lo, ext, fbo):
    _run(handler, np.asarray(lo), ext, fbo, synth.voronoi_polygons(40, seed=5, box=ext, verts_per_poly=30, jitter=5.0))


@pytest.mark.parametrize("lo,ext,fbo", [(38799352.0, 6547.0, 1176), (54720284.0, 6241.0, 2055), (50627588.0, 7458.0, 784),
                                        (60792624.0, 4212.0, 685), (53300116.0, 4468.0, 752), (40853684.0, 8358.0, 1197)])
def test_rim(handler, lo, ext, fbo):
    """Points four metres (pixels) off the canvas that fp32 puts on it, in
    extents where the coarse cells end right there; strips up to the rim."""
    x = np.linspace(0.0, ext, 9)
    strips = np.concatenate([[(a, 0), (b, 0), (b, ext), (a, ext)] for a, b in zip(x[:-1], x[1:])])
    _run(handler, np.asarray((lo, lo)), ext, fbo, (strips, 4 * np.arange(9, dtype=np.int32)))


@pytest.mark.parametrize("lo,ext,cell,fbo", [(37861176.0, 3417.0, 0.9, 1675), (39100696.0, 5340.0, 0.6, 1045),
                                             (41181008.0, 4921.0, 0.7, 915)])
def test_rim_rows_are_not_skipped(handler, lo, ext, cell, fbo):
    """Whole zones of rows four metres off the canvas that fp32 puts on it, alone
    and in a fused batch."""
    x = np.linspace(0.0, ext, 9)
    strips = np.concatenate([[(a, 0), (b, 0), (b, ext), (a, ext)] for a, b in zip(x[:-1], x[1:])])
    verts = (strips + lo).astype(np.float32)
    pidx = 4 * np.arange(9, dtype=np.int32)
    rng = np.random.default_rng(fbo)
    y = rng.uniform(lo, lo + ext, 50_000)
    xy = np.r_[np.c_[np.full(20_000, lo - 4.0), y[:20_000]], np.c_[np.full(20_000, lo + ext + 4.0), y[20_000:40_000]],
               np.c_[rng.uniform(lo, lo + ext, 10_000), y[40_000:]]].astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setCellSize(cell)
    handler.max_fbo_size = fbo
    want = oracle.raster_join(xy, verts, pidx, cell, max_res=fbo)[0]
    assert want.sum() > 15_000
    try:
        for flag in (0, rj.FLAG_FLAT_CANVAS, rj.FLAG_FORCE_CANVAS, rj.FLAG_TIERED_CANVAS):
            handler.flags = flag
            np.testing.assert_array_equal(handler.execute(rj.RasterJoinFn).count, want)
        got = handler.execute_batch([handler.make_query(rj.RasterJoinFn)] * 2, [None] * 2, flags=rj.BATCH_FUSE_ALL)[0]
        for g in got:
            np.testing.assert_array_equal(g.count, want)
    finally:
        handler.flags = 0
        handler.max_fbo_size = 8192
