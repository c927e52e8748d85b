"""Hybrid canvases wider than 65,536 pixels: the polygon pass over the point
canvas (overlapping polygons) counts and sums like the oracle."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [65535, 65536, 131075])
@pytest.mark.parametrize("nv", [9, 400])
def test_hybrid_columns_past_16_bits(handler, width, nv):
    rng = np.random.default_rng(width + nv)
    polys = [np.array([[0.0, 0.0], [40.0, 0.0], [40.0, 70.0]]), np.array([[width, 70.0], [width - 30.0, 70.0], [width, 0.0]])]
    for c in np.r_[rng.uniform(100, width - 100, 20), rng.uniform(width - 600, width - 100, 20)]:
        ang = np.sort(rng.uniform(0, 2 * np.pi, nv))
        polys.append(np.c_[c, 35.0] + rng.uniform(5, 34, (nv, 1)) * np.c_[3 * np.cos(ang), np.sin(ang)])
    verts = np.concatenate(polys).astype(np.float32)
    pidx = np.r_[0, np.cumsum([len(p) for p in polys])].astype(np.int32)
    xy = np.c_[np.r_[rng.uniform(0, width, 50_000), rng.uniform(width - 800, width, 50_001)], rng.uniform(0, 70, 100_001)]
    xy = xy.astype(np.float32)
    val = rng.uniform(-50, 90, len(xy)).astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.add_column(2, rj.Float, val)
    dh.setPolygons(verts, pidx)
    dh.setAggregation(rj.Sum, 2)
    handler.setDataHandler(dh)
    handler.setPolyIndexResolution(256)
    handler.hybrid_canvas = width
    handler.flags = rj.FLAG_FORCE_CANVAS
    f = oracle.Columns({2: (oracle.Float, val)}).filt([], aggr_attrib=2)
    want = oracle.hybrid_join(xy, verts, pidx, 256, f=f)
    try:
        got = handler.execute(rj.HybridJoinFn)
    finally:
        handler.hybrid_canvas = 0
        handler.flags = 0
    np.testing.assert_array_equal(got.count, want[0])
    # the oracle adds in fp64: 1e-6 covers its order of summation
    np.testing.assert_allclose(got.sum, want[1], rtol=1e-6, atol=1e-6 * max(1.0, float(np.abs(want[1]).max())))
    assert want[0][2:].min() > 0
