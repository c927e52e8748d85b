"""Tiered canvases whose bands of 16 rows hold about as many edges as a warp
stages: whole (112), as vertex numbers (448), or not at all (more)."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj

pytestmark = pytest.mark.gpu

SIDE = 4200.0


def _comb(x, y, teeth, step, height):
    """A comb standing on y whose teeth end inside one band of rows; 2 * teeth
    edges there and two sides."""
    k = np.arange(2 * teeth + 1)
    top = np.c_[x + step * k, y + height + np.where(k % 2 == 1, 9.3, 0.6)]
    return np.r_[top, [[x + step * 2 * teeth, y], [x, y]]]


@pytest.mark.parametrize("teeth", [(54, 55, 56, 57), (127, 128, 129, 130), (221, 222, 223, 224, 225, 226), (300, 700)])
@pytest.mark.parametrize("overlap", [False, True])
def test_edges_of_a_band(handler, teeth, overlap):
    polys = []
    for i, t in enumerate(teeth):
        step = 3900.0 / (2 * t)
        polys.append(_comb(60.0 + 7 * i, 100.0 + 350.0 * i, t, step, 40.0 + i))
        if overlap:
            polys.append(_comb(75.0 + 7 * i, 110.0 + 350.0 * i, t, step, 40.0 + i))
    polys += [np.array([[0.0, 0.0], [5.0, 0.0], [5.0, 5.0]]), np.array([[SIDE, SIDE], [SIDE - 5, SIDE], [SIDE, SIDE - 5]])]
    verts = np.concatenate(polys).astype(np.float32)
    pidx = np.r_[0, np.cumsum([len(p) for p in polys])].astype(np.int32)
    rng = np.random.default_rng(sum(teeth))
    xy = verts[rng.integers(0, len(verts), 150_000)] + rng.normal(0, [15.0, 6.0], (150_000, 2))
    xy = np.r_[xy, rng.uniform(0, SIDE, (50_001, 2))].astype(np.float32)
    val = rng.uniform(-50, 90, len(xy)).astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.add_column(2, rj.Float, val)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setCellSize(1.0)
    handler.flags = rj.FLAG_TIERED_CANVAS
    f = oracle.Columns({2: (oracle.Float, val)}).filt([], aggr_attrib=2)
    c, s, b = oracle.raster_join(xy, verts, pidx, 1.0, f=f, bounds=True)
    try:
        got = handler.execute(rj.RasterJoinBoundFn)
        np.testing.assert_array_equal(got.count, c)
        np.testing.assert_array_equal(got.bounds, b)
        dh.setAggregation(rj.Sum, 2)
        for flag in (0, rj.FLAG_FORCE_CANVAS):
            handler.flags = rj.FLAG_TIERED_CANVAS | flag
            got = handler.execute(rj.RasterJoinFn)
            np.testing.assert_array_equal(got.count, c)
            # the oracle adds in fp64: 1e-6 covers its order of summation
            np.testing.assert_allclose(got.sum, s, rtol=1e-6, atol=1e-6 * max(1.0, float(np.abs(s).max())))
    finally:
        handler.flags = 0
    assert c.sum() > 50_000 and b.any()
