"""Buffers that a prepared query's graph reads stay its own while other queries
run: a cached grid rebuilt at another resolution or for another polygon set,
scratch outgrown by a larger query, and all of it given back with the plan."""
import numpy as np
import pytest

import oracle
import rasterjoin as rj
from rasterjoin import synth

pytestmark = pytest.mark.gpu

N = 60_001


@pytest.fixture(scope="module")
def sets():
    a = synth.voronoi_polygons(260, seed=20261203)
    b = synth.star_polygons(700, seed=9, vmin=8, vmax=120, rmin=400, rmax=4000)
    return a, b


def _table(h, verts, pidx):
    xy = synth.points(N, seed=61)["xy"]
    dh = rj.DataHandler()
    dh.add_column(1, rj.Location, xy)
    dh.setPolygons(verts, pidx)
    h.setDataHandler(dh)
    h.setCellSize(100.0)
    h.setPolyIndexResolution(256)
    return xy


@pytest.fixture
def own(built):
    h = rj.GLHandler()
    yield h
    h.close()


@pytest.mark.parametrize("fn,flags", [(rj.HybridJoinFn, 0), (rj.IndexJoinFn, 0), (rj.IndexJoinFn, rj.FLAG_NO_CELL_CLASSIFY)])
def test_grid_rebuilt_between_replays(own, sets, fn, flags):
    """Coarser, finer and back, through both joins, and fresh on every call."""
    verts, pidx = sets[0]
    xy = _table(own, verts, pidx)
    want = oracle.index_join(xy, verts, pidx, 256)[0]
    own.flags = flags
    plan = own.prepare(fn)
    try:
        for other, res in ((rj.IndexJoinFn, 256), (rj.IndexJoinFn, 40), (rj.HybridJoinFn, 500), (fn, 7), (fn, 256)):
            for fl in (flags, flags | rj.FLAG_NO_CACHE):
                own.flags = fl
                own.setPolyIndexResolution(res)
                own.execute(other)
                np.testing.assert_array_equal(plan.execute().count, want)
    finally:
        plan.close()


@pytest.mark.parametrize("fn,flags", [(rj.HybridJoinFn, 0), (rj.IndexJoinFn, 0), (rj.IndexJoinFn, rj.FLAG_NO_CELL_CLASSIFY)])
def test_another_set_between_replays(own, sets, fn, flags):
    """Plans of two sets, the other one with more polygons; each replays on the
    grid it was captured with."""
    (va, pa), (vb, pb) = sets
    xy = _table(own, va, pa)
    want = [oracle.index_join(xy, v, p, 256)[0] for v, p in sets]
    own.flags = flags
    other = own.polyset(vb, pb)
    plans = []
    try:
        plans.append(own.prepare(fn))
        own.usePolySet(other)
        own.execute(fn)
        plans.append(own.prepare(fn))
        for k in (0, 1, 0, 1):
            own.usePolySet(other if k else None)
            np.testing.assert_array_equal(plans[k].execute().count, want[k])
            own.execute(fn)
            np.testing.assert_array_equal(plans[k].execute().count, want[k])
    finally:
        for p in plans:
            p.close()
        own.usePolySet(None)
        other.close()


@pytest.mark.parametrize("fn", [rj.RasterJoinFn, rj.RasterJoinBoundFn, rj.HybridJoinFn])
def test_scratch_outgrown_under_a_plan(own, sets, fn):
    verts, pidx = sets[0]
    _table(own, verts, pidx)
    want = own.execute(fn)
    plan = own.prepare(fn)
    try:
        for cell, canvas in ((25.0, 4096), (10.0, 8000)):
            own.setCellSize(cell)
            own.hybrid_canvas = canvas
            own.execute(fn)
            got = plan.execute()
            np.testing.assert_array_equal(got.count, want.count)
            if fn == rj.RasterJoinBoundFn:
                np.testing.assert_array_equal(got.bounds, want.bounds)
    finally:
        plan.close()


def test_buffers_are_given_back(built, sets):
    """A plan per round, each holding a grid of its own (10 MB and more): under
    a budget of 400 MB this only fits when a closed plan's buffers are freed,
    also while an older plan lives on."""
    verts, pidx = sets[0]
    h = rj.GLHandler(gpu_mem_mb=400)
    try:
        _table(h, verts, pidx)
        keep = h.prepare(rj.RasterJoinFn)
        want = h.execute(rj.RasterJoinFn).count
        for k in range(40):
            h.setPolyIndexResolution(256)
            plan = h.prepare(rj.IndexJoinFn)
            h.setPolyIndexResolution(250 + k % 2)
            h.execute(rj.IndexJoinFn)
            plan.execute()
            plan.close()
        np.testing.assert_array_equal(keep.execute().count, want)
        keep.close()
    finally:
        h.close()
