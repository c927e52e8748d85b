"""Counts through bins over more points than one round takes (2^27): three
rounds, the last one odd, four filter columns, and rows in order of x, so that
the zone map skips most rows of some chunks and all of others.  The rows that
pass the filters go to the oracle."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu

BINS = 6
N = (1 << 28) + 32769


def test_three_rounds(built):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(7)
    xy = torch.empty((N, 2), device="cuda")
    x = torch.arange(N, device="cuda", dtype=torch.float64)
    x.mul_(2.0 / (1 << 28)).frac_().mul_(synth.BOX)     # two sweeps, then some of a third
    xy[:, 0] = x
    del x
    xy[:, 1] = torch.rand(N, generator=g, device="cuda") * synth.BOX
    xy[1 << 28:] = torch.rand((N - (1 << 28), 2), generator=g, device="cuda") * 5000.0 + 12000.0
    cols = [torch.randint(0, 100, (N,), generator=g, device="cuda", dtype=torch.int32) for _ in range(4)]
    ok = torch.ones(N, dtype=torch.bool, device="cuda")
    for c in cols:
        ok &= c < 40
    kept = xy[ok].cpu().numpy()
    assert kept.shape[0] > 6_000_000 and int(ok[1 << 28:].sum()) > 500
    del ok
    verts, pidx = synth.star_polygons(60, seed=43, box=9000.0, vmin=8, vmax=60, rmin=300, rmax=2000)
    verts = (verts + np.float32(10000.0)).astype(np.float32)
    h = rj.GLHandler()
    try:
        dh = rj.DataHandler()
        dh.declare(1, rj.Location)
        for k in range(4):
            dh.declare(2 + k, rj.Int)
        dh.setQueryConstraints([(2 + k, rj.LT, 40) for k in range(4)])
        h.attachDevice([(1, rj.Location, xy.data_ptr())] + [(2 + k, rj.Int, c.data_ptr()) for k, c in enumerate(cols)], N, 1)
        ps = h.polyset(verts, pidx)
        h.usePolySet(ps)
        h.dataHandler = dh
        h.setCellSize(10.0)
        h.flags = rj.FLAG_FORCE_CANVAS | rj.FLAG_FLAT_CANVAS
        qs = [(fn, h.make_query(fn)) for fn in (rj.RasterJoinFn, rj.RasterJoinBoundFn)]
        h.dataHandler = None
        torch.cuda.synchronize()
        h.setTuning(rj.TUNE_COUNT_SHAPE, BINS)
        got = []
        for fn, q in qs:
            got.append(h.execute(fn, q))
            assert h.getTuning(rj.TUNE_COUNT_SHAPE) == BINS
        ps.close()
    finally:
        h.close()
    want = oracle.raster_join(kept, verts, pidx, 10.0, bounds=True)
    np.testing.assert_array_equal(got[0].count, want[0])
    np.testing.assert_array_equal(got[1].count, want[0])
    np.testing.assert_array_equal(got[1].bounds, want[2])
    assert want[0].sum() > 100_000
