"""A tuned choice is an index into the candidates of its query class: canvases of
the same octave whose block sides differ are classes of their own (the first
query on each times its candidates, which shows in the launches)."""
import numpy as np
import pytest

import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu

N = (1 << 22) + 1
TIMED = 8          # at least four candidates, each launched twice


def test_each_candidate_list_is_timed(built):
    verts, pidx = synth.voronoi_polygons(37, seed=5, verts_per_poly=24)
    h = rj.GLHandler()
    try:
        dh = rj.DataHandler()
        dh.add_column(1, rj.Location, synth.points(N, seed=71)["xy"])
        dh.setPolygons(verts, pidx)
        h.setDataHandler(dh)
        h.flags = rj.FLAG_FLAT_CANVAS
        ext = float(max(verts.max(0) - verts.min(0)))
        counts = []
        for size in (4096, 4160):   # blocks of 16 and 32 pixels, of 32 and 64
            h.setCellSize(ext / (size - 0.5))
            launches = []
            for _ in range(2):
                counts.append(h.execute(rj.RasterJoinFn).count)
                launches.append(h.timings()["kernel_launches"])
            assert launches[0] - launches[1] >= TIMED
        assert abs(int(counts[0].sum()) - N) < N // 1000
        np.testing.assert_array_equal(counts[0], counts[1])
        np.testing.assert_array_equal(counts[2], counts[3])
    finally:
        h.close()
