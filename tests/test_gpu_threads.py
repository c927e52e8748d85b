"""Contexts on several threads: queries whose passes run the same kernel with
different amounts of shared memory, at the same time."""
import ctypes as C
import threading

import numpy as np
import pytest

import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu

SIDES = (2650, 2700, 2800, 3000, 3300, 3600, 4000, 4050)   # 54 to 128 KB of block codes


def test_shared_memory_of_one_kernel(built):
    verts, pidx = synth.voronoi_polygons(40, seed=5, verts_per_poly=30)
    xy = synth.points(1001, seed=81)["xy"]
    ext = float(max(verts.max(0) - verts.min(0)))
    wrong = []

    def work(side):
        h = rj.GLHandler()
        try:
            dh = rj.DataHandler()
            dh.add_column(1, rj.Location, xy)
            dh.setPolygons(verts, pidx)
            h.setDataHandler(dh)
            h.setCellSize(ext / (side - 0.5))
            h.flags = rj.FLAG_FLAT_CANVAS
            h.setTuning(rj.TUNE_COUNT_SHAPE, 0)
            h.setTuning(rj.TUNE_COUNT_BLOCK_SHIFT, 4)
            want = h.execute(rj.RasterJoinFn).count
            q = h.make_query(rj.RasterJoinFn)
            for k in range(6000):
                rc = h.lib.rj_execute(h.ctx, C.byref(q), None)
                if rc or h.getTuning(rj.TUNE_COUNT_SHAPE) != 0:
                    wrong.append((side, k, rc))
            np.testing.assert_array_equal(h.execute(rj.RasterJoinFn).count, want)
        except Exception as e:   # noqa: BLE001 - reported by the test's own thread
            wrong.append((side, e))
        finally:
            h.close()

    threads = [threading.Thread(target=work, args=(side,)) for side in SIDES]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
