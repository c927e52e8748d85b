"""Sides of the one-tile label pass's blocks at the limits of its code map: a map
of 128 KB and one entry, larger ones when the side is forced, and a forced side
whose map does not fit (the generic pass)."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,shift,lean", [(4080, 4, True), (4081, 4, True), (4096, 4, True), (4097, 4, True), (4500, 4, True),
                                            (6000, 4, False), (8192, 5, True), (8161, 5, True), (8192, 4, False)])
def test_forced_side(handler, res, shift, lean):
    verts, pidx = synth.voronoi_polygons(40, seed=5, verts_per_poly=30)
    xy = synth.points(100_001, seed=res)["xy"]
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    ext = float(max(verts.max(0) - verts.min(0)))
    handler.setCellSize(ext / (res - 0.5))
    handler.setTuning(rj.TUNE_COUNT_BLOCK_SHIFT, shift)
    handler.flags = rj.FLAG_FLAT_CANVAS
    try:
        got = handler.execute(rj.RasterJoinFn)
        ran = handler.getTuning(rj.TUNE_COUNT_BLOCK_SHIFT)
    finally:
        handler.setTuning(rj.TUNE_COUNT_BLOCK_SHIFT, -1)
        handler.flags = 0
    np.testing.assert_array_equal(got.count, oracle.raster_join(xy, verts, pidx, ext / (res - 0.5))[0])
    assert ran == (shift if lean else -1)


@pytest.mark.parametrize("cell,filters", [(100.0, False), (100.0, True), (5.0, False)])
def test_shape_indices_past_the_shapes(handler, cell, filters):
    """Indices that older libraries had shapes for still give a lean pass; others
    are refused."""
    verts, pidx = synth.voronoi_polygons(40, seed=5, verts_per_poly=30)
    pts = synth.points(100_001, seed=82, columns=True)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, pts["xy"])
    dh.add_column(4, rj.Int, pts["f1"])
    dh.setPolygons(verts, pidx)
    if filters:
        dh.setQueryConstraints([(4, rj.GTE, 2)])
    handler.setDataHandler(dh)
    handler.setCellSize(cell)
    try:
        want = handler.execute(rj.RasterJoinFn).count
        for shape in range(11):
            handler.setTuning(rj.TUNE_COUNT_SHAPE, shape)
            np.testing.assert_array_equal(handler.execute(rj.RasterJoinFn).count, want)
            ran = handler.getTuning(rj.TUNE_COUNT_SHAPE)
            assert ran == shape if shape < 3 else ran >= 0
        for shape in (-2, 11):
            with pytest.raises(rj.RJError):
                handler.setTuning(rj.TUNE_COUNT_SHAPE, shape)
    finally:
        handler.setTuning(rj.TUNE_COUNT_SHAPE, -1)
