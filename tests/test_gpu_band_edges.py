"""Polygon passes over point canvases (rj_band_kernels.cu): nearly horizontal
edges, on which the outline clip's rounding of y moves an accepted pixel by up
to a pixel along the row; rows with more crossings than a warp holds; polygons
thinner than a pixel and partly off the canvas; sums.  Counts, sums and error
bounds equal the oracle's on flat and tiered canvases, one tile and several."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj

pytestmark = pytest.mark.gpu

BOX = 6000.0


def flat_edges():
    """Quadrilaterals whose long edges fall 5e-4 to 2e-3 per pixel, high on the
    canvas (coordinates above 4096 have a unit in the last place of 2^-11), and
    points around the places where those edges cross rows of pixels."""
    rng = np.random.default_rng(17)
    polys, pts = [], []
    for _ in range(120):
        x0, y0 = rng.uniform(100, 4500), rng.uniform(4200, 5900)
        w, s = rng.uniform(300, 1400), rng.uniform(5e-4, 2e-3) * rng.choice([-1, 1])
        polys.append(np.array([[x0, y0], [x0 + w, y0 + s * w], [x0 + w, y0 + s * w + 30], [x0, y0 + 40]], np.float32))
        for row in range(int(np.floor(min(y0, y0 + s * w))), int(np.ceil(max(y0, y0 + s * w))) + 1):
            x = x0 + (row - y0) / s
            if x0 <= x <= x0 + w:
                g = np.mgrid[-4:5, -2:3].reshape(2, -1).T + 0.5
                pts.append(np.floor([x, row]) + g)
    return polys, np.concatenate(pts)


def combs():
    """A comb of 700 teeth (over 512 crossings a row), slivers thinner than a
    pixel in either direction, and a frame reaching past the others' bounds."""
    k = np.arange(1401)
    teeth = np.c_[50.0 + 4.0 * k, 3000.0 + np.where(k % 2 == 1, 60.3, 0.3)]
    polys = [np.r_[teeth, [[5650.0, 2980.7], [50.0, 2980.7]]],
             np.array([[10.2, 10.2], [10.7, 10.2], [10.7, 5990.0], [10.2, 5990.0]]),
             np.array([[10.0, 20.3], [5990.0, 20.3], [5990.0, 20.45], [10.0, 20.45]]),
             np.array([[1.0, 1.0], [5999.0, 1.0], [5999.0, 5999.0], [3000.0, 4000.0], [1.0, 5999.0]])]
    rng = np.random.default_rng(3)
    pts = np.r_[rng.uniform(0, BOX, (40_000, 2)), np.c_[rng.uniform(40, 5660, 40_000), rng.uniform(2978, 3062, 40_000)],
                np.c_[rng.uniform(9, 12, 5000), rng.uniform(0, BOX, 5000)],
                np.c_[rng.uniform(0, BOX, 5000), rng.uniform(19, 22, 5000)]]
    return [p.astype(np.float32) for p in polys], pts


@pytest.mark.parametrize("shape", [flat_edges, combs])
@pytest.mark.parametrize("fbo", [8192, 2100])
@pytest.mark.parametrize("cell", [1.0, 1.7])
def test_band_passes_match_oracle(handler, shape, fbo, cell):
    polys, pts = shape()
    corner = [np.array([[0, 0], [3, 0], [3, 3]], np.float32), np.array([[BOX, BOX], [BOX - 3, BOX], [BOX, BOX - 3]], np.float32)]
    polys = polys + corner                                   # the canvas spans the box
    verts = np.concatenate(polys)
    pidx = np.r_[0, np.cumsum([len(p) for p in polys])].astype(np.int32)
    xy = pts.astype(np.float32)
    a = np.random.default_rng(5).lognormal(2.5, 0.8, len(xy)).astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.add_column(2, rj.Float, a)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setCellSize(cell)
    handler.max_fbo_size = fbo
    f = oracle.Columns({2: (oracle.Float, a)}).filt([], aggr_attrib=2)
    c, s, b = oracle.raster_join(xy, verts, pidx, cell, f=f, max_res=fbo, bounds=True)
    try:
        for flag in (rj.FLAG_FLAT_CANVAS, rj.FLAG_TIERED_CANVAS):
            handler.flags = flag
            dh.setAggregation(rj.Count, -1)
            got = handler.execute(rj.RasterJoinBoundFn)
            np.testing.assert_array_equal(got.count, c)
            np.testing.assert_array_equal(got.bounds, b)
            handler.flags = flag | rj.FLAG_FORCE_CANVAS
            dh.setAggregation(rj.Sum, 2)
            got = handler.execute(rj.RasterJoinFn)
            np.testing.assert_array_equal(got.count, c)
            np.testing.assert_allclose(got.sum, s, rtol=1e-6, atol=1e-6)
    finally:
        handler.flags = 0
        handler.max_fbo_size = 8192
    assert b[:2 * len(polys)].any()


@pytest.mark.parametrize("nv", [130, 700, 2500])
@pytest.mark.parametrize("fbo", [8192, 311])
def test_jagged_outlines_match_oracle(handler, nv, fbo):
    """Rings that cross a row up to thousands of times (rows kept as bitmaps),
    beside plain ones in the same bands: counts, sums and error bounds."""
    rng = np.random.default_rng(nv)
    polys = []
    for k in range(6):
        ang = np.sort(rng.uniform(0, 2 * np.pi, nv if k % 3 else 9))
        rad = rng.uniform(5, 330, len(ang))
        polys.append(np.c_[500 + 90 * k + rad * np.cos(ang), 500 + 40 * (k % 2) + rad * np.sin(ang)].astype(np.float32))
    verts = np.concatenate(polys)
    pidx = np.r_[0, np.cumsum([len(p) for p in polys])].astype(np.int32)
    xy = rng.uniform(100, 1400, (200_001, 2)).astype(np.float32)
    val = rng.uniform(-50, 90, len(xy)).astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.add_column(2, rj.Float, val)
    dh.setPolygons(verts, pidx)
    dh.setAggregation(rj.Avg, 2)
    handler.setDataHandler(dh)
    handler.setCellSize(1.0)
    handler.max_fbo_size = fbo
    handler.flags = rj.FLAG_FORCE_CANVAS | rj.FLAG_FLAT_CANVAS
    f = oracle.Columns({2: (oracle.Float, val)}).filt([], aggr_attrib=2)
    try:
        got = handler.execute(rj.RasterJoinFn)
        want = oracle.raster_join(xy, verts, pidx, 1.0, f=f, max_res=fbo)
        np.testing.assert_array_equal(got.count, want[0])
        np.testing.assert_allclose(got.sum, want[1], rtol=1e-6, atol=1e-9 * max(1.0, float(np.abs(want[1]).max())))
        dh.setAggregation(rj.Count, -1)
        handler.setDataHandler(dh)
        bnd = handler.execute(rj.RasterJoinBoundFn)
        want = oracle.raster_join(xy, verts, pidx, 1.0, max_res=fbo, bounds=True)
        np.testing.assert_array_equal(bnd.count, want[0])
        np.testing.assert_array_equal(bnd.bounds, want[2])
    finally:
        handler.flags = 0
        handler.max_fbo_size = 8192
