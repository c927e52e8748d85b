"""The classified grid of the exact tests, built a pair of cell and polygon per
warp or per lane (polygons of more than 512 vertices by the warp): outlines on
both sides of that limit, side by side in one set so that warps hold pairs of
several polygons, coarse and fine grids; index and hybrid counts equal the
oracle's, on points crowded along the outlines."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj

pytestmark = pytest.mark.gpu

# many edges per pair: a warp per pair; few: a lane per pair, but for the rings
# of more than 512
SIZES = [3, 4, 7, 8, 9, 100, 511, 512, 513, 640, 1200, 5, 31, 33, 2000, 3]
SMALL = [3, 4, 7, 8, 9, 100, 32, 64, 513, 65, 512, 5, 31, 33, 3, 3]


def _set(overlap, sizes=SIZES):
    rng = np.random.default_rng(17)
    polys = []
    for i, n in enumerate(sizes):
        cx, cy = 500.0 + 1000.0 * (i % 4), 500.0 + 1000.0 * (i // 4)
        ang = np.sort(rng.uniform(0, 2 * np.pi, n)) if n > 4 else 2 * np.pi * (np.arange(n) + 0.3) / n
        rad = rng.uniform(150.0, 460.0, n) * (1.6 if overlap else 1.0)
        polys.append(np.c_[cx + rad * np.cos(ang), cy + rad * np.sin(ang)])
    v = np.concatenate(polys).astype(np.float32)
    return v, np.r_[0, np.cumsum(sizes)].astype(np.int32)


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("res", [1, 5, 64, 300, 500])
@pytest.mark.parametrize("sizes", [SIZES, SMALL])
def test_joins_match_oracle(handler, overlap, res, sizes):
    verts, pidx = _set(overlap, sizes)
    rng = np.random.default_rng(18)
    on = verts[rng.integers(0, len(verts), 100_000)] + rng.normal(0, 2.0, (100_000, 2))
    xy = np.r_[rng.uniform(-300, 4300, (150_001, 2)), on].astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setPolyIndexResolution(res)
    got = handler.execute(rj.IndexJoinFn)
    np.testing.assert_array_equal(got.count, oracle.index_join(xy, verts, pidx, res)[0])
    got = handler.execute(rj.HybridJoinFn)
    np.testing.assert_array_equal(got.count, oracle.hybrid_join(xy, verts, pidx, res)[0])


@pytest.mark.parametrize("canvas", [1000, 1001, 1004, 1021, 33])
def test_label_map_widths(handler, canvas):
    """Label maps of the hybrid canvas whose rows do and do not allow 16-byte
    loads (finishing, block codes)."""
    verts, pidx = _set(False)
    xy = np.random.default_rng(19).uniform(-300, 4300, (200_001, 2)).astype(np.float32)
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setPolyIndexResolution(64)
    handler.hybrid_canvas = canvas
    try:
        got = handler.execute(rj.HybridJoinFn)
    finally:
        handler.hybrid_canvas = 0
    np.testing.assert_array_equal(got.count, oracle.hybrid_join(xy, verts, pidx, 64)[0])
