"""Counts onto the point canvas through bins (points ordered by 128 x 128-pixel
bin, then counted in shared memory): counts and error bounds equal the oracle's
on canvases of one bin up to some hundred bins with ragged edges, on tables
around the 16,384 points ordered at a time, with every number of filter
columns, with points outside the canvas, and with nearly all points in a few
pixels (a bin cut into parts, runs longer than a warp)."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu

BINS = 6
BOX = 40000.0
SPECIALS = np.array([[np.nan, 10.0], [10.0, np.nan], [np.inf, 5.0], [-np.inf, 5.0], [1e30, 1e30], [-1e30, 3.0],
                     [0.0, 0.0], [BOX, BOX], [0.0, 39999.996], [39999.996, 0.0], [-0.004, 20000.0]], np.float32)


@pytest.fixture(scope="module")
def stars():
    return synth.star_polygons(40, seed=43, vmin=8, vmax=60, rmin=1000, rmax=6000)


def _points(n, crowded, seed=51):
    pts = synth.points(n, seed=seed, columns=True)
    rng = np.random.default_rng(seed)
    xy = pts["xy"].copy()
    if crowded:   # 60 % within 40 m, 20 % within 2 km of a polygon's middle
        m = int(n * 0.6)
        xy[:m] = np.float32([17000.0, 23000.0]) + rng.uniform(0, 40, (m, 2)).astype(np.float32)
        xy[m:m + n // 5] = rng.normal([17000.0, 23000.0], 2000.0, (n // 5, 2)).astype(np.float32)
        xy = xy[rng.permutation(n)]
    k = min(len(SPECIALS), n // 4)
    xy[rng.choice(n, k, replace=False)] = SPECIALS[:k]
    pts["xy"] = xy
    return pts


def _run(handler, pts, stars, cell, ncols):
    verts, pidx = stars
    cons = [(4, rj.GT, 2), (3, rj.LT, 60.0), (2, rj.GT, synth.T0 + synth.YEAR // 3), (5, rj.LT, 8)][:ncols]
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, pts["xy"])
    dh.add_column(2, rj.Uint, pts["t"])
    dh.add_column(3, rj.Float, pts["a"])
    dh.add_column(4, rj.Int, pts["f1"])
    dh.add_column(5, rj.Int, pts["f1"])
    dh.setPolygons(verts, pidx)
    if cons:
        dh.setQueryConstraints(cons)
    handler.setDataHandler(dh)
    handler.setCellSize(cell)
    f = None
    if cons:
        cols = oracle.Columns({2: (oracle.Uint, pts["t"]), 3: (oracle.Float, pts["a"]), 4: (oracle.Int, pts["f1"]),
                               5: (oracle.Int, pts["f1"])})
        f = cols.filt(cons)
    want = oracle.raster_join(pts["xy"], verts, pidx, cell, f=f, bounds=True)
    handler.setTuning(rj.TUNE_COUNT_SHAPE, BINS)
    handler.flags = rj.FLAG_FORCE_CANVAS | rj.FLAG_FLAT_CANVAS
    try:
        got = handler.execute(rj.RasterJoinFn)
        ran = handler.getTuning(rj.TUNE_COUNT_SHAPE)
        bnd = handler.execute(rj.RasterJoinBoundFn)
    finally:
        handler.setTuning(rj.TUNE_COUNT_SHAPE, -1)
        handler.flags = 0
    assert ran == BINS
    np.testing.assert_array_equal(got.count, want[0])
    np.testing.assert_array_equal(bnd.count, want[0])
    np.testing.assert_array_equal(bnd.bounds, want[2])


@pytest.mark.parametrize("cell", [400.0, 77.0, 10.0])      # 1, 25 and 1,024 bins
@pytest.mark.parametrize("crowded", [False, True])
def test_canvas_sizes(handler, stars, cell, crowded):
    _run(handler, _points(1_500_001, crowded), stars, cell, 0)


@pytest.mark.parametrize("n", [1, 2, 16383, 16384, 16385, 100_000])
def test_table_sizes(handler, stars, n):
    _run(handler, _points(n, False), stars, 40.0, 0)


@pytest.mark.parametrize("ncols", [1, 2, 3, 4])
def test_filter_columns(handler, stars, ncols):
    _run(handler, _points(300_001, False), stars, 40.0, ncols)
