"""The bins' scratch (two bytes a point) is held only where counting through bins
is the kept choice: 2^26 points onto 64 x 64 pixels, where copies of the canvas
in shared memory win, and onto 4000 x 4000, whichever wins there."""
import numpy as np
import pytest

import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu

BINS = 6
N = 1 << 26


@pytest.mark.parametrize("cell,wins", [(synth.BOX / 64, False), (10.0, None)])
def test_scratch_follows_the_choice(built, cell, wins):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(5)
    xy = torch.rand((N, 2), generator=g, device="cuda") * synth.BOX
    verts, pidx = synth.star_polygons(40, seed=43, vmin=8, vmax=60, rmin=1000, rmax=6000)
    h = rj.GLHandler()
    try:
        dh = rj.DataHandler()
        dh.declare(1, rj.Location)
        h.attachDevice([(1, rj.Location, xy.data_ptr())], N, 1)
        corner = np.float32([[0, 0], [9, 0], [9, 9], [synth.BOX, synth.BOX], [synth.BOX - 9, synth.BOX], [synth.BOX, synth.BOX - 9]])
        ps = h.polyset(np.r_[verts, corner], np.r_[pidx, pidx[-1] + 3, pidx[-1] + 6])
        h.usePolySet(ps)
        h.dataHandler = dh
        h.setCellSize(cell)
        h.flags = rj.FLAG_FORCE_CANVAS | rj.FLAG_FLAT_CANVAS
        q = h.make_query(rj.RasterJoinFn)
        h.dataHandler = None
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        first = h.execute(rj.RasterJoinFn, q)
        again = h.execute(rj.RasterJoinFn, q)
        ran = h.getTuning(rj.TUNE_COUNT_SHAPE)
        taken = before - torch.cuda.mem_get_info()[0]
        np.testing.assert_array_equal(first.count, again.count)
        assert wins is None or (ran == BINS) == wins
        # 64 MB of canvas and small change; the bins would take 2 * N bytes more
        assert (taken >= 2 * N) == (ran == BINS), taken
        ps.close()
    finally:
        h.close()
