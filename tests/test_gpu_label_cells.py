"""Label pass over coarse cells (rj_label_core.cuh): counts and sums equal the
oracle's where the cell grid can go wrong -- canvases away from the origin
(where fp32 rounding reaches whole pixels), points on cell edges and tile
seams, cells of one pixel row, one polygon, odd and tiny tables, and filter
columns given in any order of types."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu


def _points(n, lo, ext, cell, seed):
    """Random locations over the box and beyond, and locations on and beside
    multiples of 4, 16 and 64 pixels."""
    rng = np.random.default_rng(seed)
    xy = rng.uniform(-0.05, 1.05, (n, 2)) * ext
    k = n // 3
    step = rng.choice([4.0, 16.0, 64.0], (k, 2)) * cell
    xy[:k] = np.rint(xy[:k] / step) * step + rng.choice([0.0, 1e-3, -1e-3, 0.5, -0.5], (k, 2)) * cell
    xy = (xy + np.asarray(lo)).astype(np.float32)
    xy[-4:] = [[np.nan, lo[1]], [np.inf, lo[1]], [-np.inf, np.nan], [3e38, -3e38]]
    return xy


@pytest.mark.parametrize("lo", [(0.0, 0.0), (-1234.5, 777.25), (500000.0, 4100000.0), (16000000.0, 16000000.0)])
@pytest.mark.parametrize("nsites,n,fbo", [(1, 5, 8192), (40, 100_001, 8192), (40, 100_000, 1700), (3, 33_333, 300)])
@pytest.mark.parametrize("tiered", [False, True])
def test_cells_match_oracle(handler, lo, nsites, n, fbo, tiered):
    ext, cell = 6000.0, 1.4 if tiered else 7.0
    verts, pidx = synth.voronoi_polygons(nsites, seed=5 + nsites, box=ext, verts_per_poly=30, jitter=5.0)
    verts = (verts.astype(np.float64) + np.asarray(lo)).astype(np.float32)
    xy = _points(n, lo, ext, cell, n)
    rng = np.random.default_rng(n)
    a = rng.lognormal(2.5, 0.8, n).astype(np.float32)
    f1 = rng.integers(-5, 5, n).astype(np.int32)
    t = rng.integers(0, 2 ** 32, n, dtype=np.uint32)
    dh = rj.DataHandler()
    for k, typ, col in ((1, rj.Location, xy), (2, rj.Float, a), (3, rj.Int, f1), (4, rj.Uint, t)):
        dh.add_column(k, typ, col)
    dh.setPolygons(verts, pidx)
    handler.setDataHandler(dh)
    handler.setCellSize(cell)
    handler.max_fbo_size = fbo
    handler.flags = rj.FLAG_TIERED_CANVAS if tiered else 0
    cols = oracle.Columns({2: (oracle.Float, a), 3: (oracle.Int, f1), 4: (oracle.Uint, t)})
    try:
        for cons, aggr in (([], None), ([(2, rj.LT, 30.0), (3, rj.GTE, -2), (4, rj.GT, 10 ** 9)], 3),
                           ([(4, rj.LTE, 3 * 10 ** 9), (2, rj.GT, 4.0)], 2), ([(3, rj.LT, 0)], None)):
            dh.setQueryConstraints(cons)
            dh.setAggregation(rj.Sum if aggr else rj.Count, aggr if aggr else -1)
            f = cols.filt(cons, aggr_attrib=aggr) if cons else None
            want_c, want_s = oracle.raster_join(xy, verts, pidx, cell, f=f, max_res=fbo)[:2]
            got = handler.execute(rj.RasterJoinFn)
            np.testing.assert_array_equal(got.count, want_c)
            if aggr:   # the oracle adds in fp64: 1e-6 covers its order of summation
                np.testing.assert_allclose(got.sum, want_s, rtol=1e-6, atol=1e-6 * max(1.0, np.abs(want_s).max()))
    finally:
        handler.max_fbo_size = 8192
        handler.flags = 0
