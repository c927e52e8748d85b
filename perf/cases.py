"""Timed cases of the join library: what a program asks of it in earnest.

Every case is a call through the Python binding (rasterjoin.GLHandler) that
mirrors the reference's join dispatcher: one join per call, a replayed plan,
a batch, or a burst of served requests.  Tables and polygons are the
benchmark configurations' shapes (a 40 x 40 km box, 80 % of the points from 8
Gaussians, Voronoi neighbourhoods or overlapping star polygons), drawn from
the seed.  Tables of up to a few million rows are loaded from host arrays, as
a program with a file would; larger ones are attached where they lie on the
GPU, as a program with a resident table would.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "raster-join_gb300"))
import rasterjoin as rj  # noqa: E402
from rasterjoin import synth, workloads  # noqa: E402

BOX, T0, YEAR = synth.BOX, synth.T0, synth.YEAR
HOST_ROWS = 4_000_000      # tables up to here are loaded from host arrays
LOC, TIME, VALUE, KIND, GRADE = 1, 2, 3, 4, 5   # attribute ids
FN = {"raster": rj.RasterJoinFn, "bounds": rj.RasterJoinBoundFn, "hybrid": rj.HybridJoinFn, "index": rj.IndexJoinFn}


def listed():
    return [
        # a first look at a small extract at the reference's default accuracy: latency and launches
        {"name": "small raster count", "call": "execute", "join": "raster", "points": 20_011, "polys": "cells",
         "npolys": 64, "cell": 100.0, "filters": 0, "avg": False, "fresh": False},
        # error bounds of a city's neighbourhoods over a month's extract (benchmark configuration 1)
        {"name": "1M error bounds 10 m", "call": "execute", "join": "bounds", "points": 1_000_000, "polys": "cells",
         "npolys": 260, "cell": 10.0, "filters": 0, "avg": False, "fresh": False},
        # a dashboard's panel, the same query over and over: a prepared plan
        {"name": "1M prepared average", "call": "prepared", "join": "raster", "points": 1_000_003, "polys": "cells",
         "npolys": 260, "cell": 10.0, "filters": 2, "avg": True, "fresh": False},
        # a filtered average over a year's table, bounded error (benchmark configuration 2 as a raster join)
        {"name": "100M raster average", "call": "execute", "join": "raster", "points": 100_000_000, "polys": "cells",
         "npolys": 260, "cell": 10.0, "filters": 4, "avg": True, "fresh": False},
        # the same query answered exactly, every polygon structure rebuilt (benchmark configuration 2)
        {"name": "100M hybrid average", "call": "execute", "join": "hybrid", "points": 100_000_000, "polys": "cells",
         "npolys": 260, "cell": 10.0, "filters": 4, "avg": True, "fresh": True},
        # ... and through the grid index, whose structures a program keeps between queries
        {"name": "100M index average", "call": "execute", "join": "index", "points": 99_999_989, "polys": "cells",
         "npolys": 260, "cell": 10.0, "filters": 4, "avg": True, "fresh": False},
        # the headline: two billion points counted at 10 m (benchmark configuration 3)
        {"name": "2B raster count 10 m", "call": "execute", "join": "raster", "points": 2_000_000_000,
         "polys": "cells", "npolys": 260, "cell": 10.0, "filters": 0, "avg": False, "fresh": True},
        # overlapping regions (catchments, user-drawn areas): the point canvas
        {"name": "500M stars 10 m", "call": "execute", "join": "raster", "points": 500_000_001, "polys": "stars",
         "npolys": 2000, "cell": 10.0, "filters": 0, "avg": False, "fresh": False},
        # the finest accuracy over a large table: the tiered canvas, labels
        {"name": "1B raster count 1 m", "call": "execute", "join": "raster", "points": 1_000_000_000,
         "polys": "cells", "npolys": 260, "cell": 1.0, "filters": 0, "avg": False, "fresh": False},
        # error bounds of overlapping regions at the finest accuracy: outlines dominate
        {"name": "200M stars bounds 1 m", "call": "execute", "join": "bounds", "points": 200_000_003,
         "polys": "stars", "npolys": 2000, "cell": 1.0, "filters": 0, "avg": False, "fresh": False},
        # a report: many queries, each with its own regions, accuracy and time window, over one table
        # (benchmark configuration 4)
        {"name": "batch of 64", "call": "batch", "points": 200_000_000, "queries": 64, "max_verts": 100_000},
        # map clients: a burst of requests with their own regions and zoom levels (benchmark configuration 5)
        {"name": "48 served requests", "call": "served", "points": 200_000_000, "queries": 48},
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    call = rng.choice(["execute"] * 7 + ["prepared", "batch", "served"])
    if call == "batch":
        return {"call": call, "points": int(log(3e5, 2e8)) | 1, "queries": int(log(2, 64)),
                "max_verts": int(log(2000, 100_000))}
    if call == "served":
        return {"call": call, "points": int(log(3e5, 2e8)) | 1, "queries": int(log(2, 48))}
    polys = rng.choice(["cells", "stars"])
    join = "raster" if call == "prepared" else rng.choice(["raster", "raster", "bounds", "hybrid", "index"])
    cell = log(10.5, 1000.0) if call == "prepared" else log(1.0, 1000.0)   # plans take no tiered canvases
    return {"call": call, "join": join, "points": int(log(1e4, 4e8)), "polys": polys,
            "npolys": int(log(16, 600) if polys == "cells" else log(1, 2000)), "cell": round(cell, 3),
            "filters": rng.randrange(5), "avg": join != "bounds" and rng.random() < 0.5,
            "fresh": rng.random() < 0.5}


# ---- inputs ----------------------------------------------------------------
def table(n, seed, names):
    """The columns `names` of a table of n rows, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda")

    out = {k: torch.empty((n, 2) if k == LOC else n, device="cuda",
                          dtype=torch.float32 if k in (LOC, VALUE) else torch.int32) for k in names}
    centres = rand(8, 2) * BOX
    step = 1 << 26
    for s in range(0, n, step):
        m = min(step, n - s)
        u = rand(m, 2) * BOX
        near = torch.randn((m, 2), generator=g, device="cuda") * 2000.0
        near += centres[torch.randint(0, 8, (m,), generator=g, device="cuda")]
        keep = (rand(m) < 0.8) & ((near >= 0) & (near < BOX)).all(1)
        p = torch.where(keep[:, None], near, u)
        out[LOC][s:s + m] = p.clamp_(0.0, math.nextafter(BOX, 0.0))
        if TIME in out:
            out[TIME][s:s + m] = torch.randint(T0, T0 + YEAR, (m,), generator=g, device="cuda", dtype=torch.int32)
        if VALUE in out:
            out[VALUE][s:s + m] = torch.exp(torch.randn(m, generator=g, device="cuda") * 0.8 + 2.5)
        for k in (KIND, GRADE):
            if k in out:
                out[k][s:s + m] = torch.randint(0, 10, (m,), generator=g, device="cuda", dtype=torch.int32)
    return out


def regions(case, seed):
    if case["polys"] == "cells":
        return synth.voronoi_polygons(case["npolys"], seed=seed)
    return workloads.star_set(np.random.default_rng(seed), case["npolys"], 20, 500, 200.0, 2000.0)


def requests(case, seed):
    """[(xy, pindex, cell, (t0, t1), avg)] of a batch or a burst, with the
    sizes of workloads.batched_queries and served_requests: how many regions,
    how fine and how long a window is the case's, where they lie the seed's."""
    sizes, places = np.random.default_rng(case["queries"]), np.random.default_rng(seed)
    n, out = case["points"], []
    for i in range(case["queries"]):
        if case["call"] == "batch":
            npolys = int(np.exp(sizes.uniform(0.0, np.log(5000.0))))
            vmin, vmax = 4, min(2000.0, max(4.0, case["max_verts"] / npolys))
            rmax = 10000.0 if npolys <= 20 else max(300.0, 10000.0 / np.sqrt(npolys / 20.0))
            cell = float(np.exp(sizes.uniform(0.0, np.log(1000.0))))
            span = int(np.exp(sizes.uniform(np.log(min(1.0, 1e4 / n)), 0.0)) * YEAR)
        else:
            npolys, vmin, vmax, rmax = int(sizes.integers(1, 51)), 8, 300, 10000.0
            cell = float(sizes.choice([1.0, 10.0, 100.0, 1000.0]))
            span = int(np.exp(sizes.uniform(np.log(workloads.HOUR), np.log(30 * workloads.DAY))))
        xy, pidx = workloads.star_set(places, npolys, vmin, vmax, 200.0, rmax)
        start = T0 + int(places.uniform(0, max(1, YEAR - span)))
        out.append((xy, pidx, cell, (start, min(start + span, T0 + YEAR - 1)), case["call"] == "batch" and bool(i % 2)))
    return out


def conditions(case):
    """Constraints and time range of a case: 1 the first half of the year, 2
    also KIND > 2, 3 also GRADE < 8, 4 also VALUE < 50."""
    cons = [(KIND, rj.GT, 2), (GRADE, rj.LT, 8), (VALUE, rj.LT, 50.0)][:max(0, case["filters"] - 1)]
    return cons, (TIME, T0, T0 + YEAR // 2) if case["filters"] else None


def columns(case):
    if case["call"] in ("batch", "served"):
        return [LOC, TIME, VALUE]
    names = [LOC, TIME, KIND, GRADE, VALUE][:case["filters"] + 1]
    return names if not case["avg"] or VALUE in names else names + [VALUE]


TYPES = {LOC: rj.Location, TIME: rj.Uint, VALUE: rj.Float, KIND: rj.Int, GRADE: rj.Int}


class Program:
    """What a user's program holds: a handler with its table and polygons."""

    def __init__(self, case, seed):
        self.case = case
        self.sets, self.plan, self.server = [], None, None
        n, names = case["points"], columns(case)
        cols = table(n, seed, names)
        self.h = rj.GLHandler()
        dh = self.dh = rj.DataHandler()
        many = case["call"] in ("batch", "served")
        if n <= HOST_ROWS and not many:
            for k in names:
                a = cols[k].cpu().numpy()
                dh.add_column(k, TYPES[k], a.view(np.uint32) if k == TIME else a)
        else:
            self.columns = cols
            torch.cuda.synchronize()
            self.h.attachDevice([(k, TYPES[k], cols[k].data_ptr()) for k in names], n, LOC)
            for k in names:
                dh.declare(k, TYPES[k])
        if many:
            # time buckets and a coarse spatial order, as for a table that serves many windows
            self.h.clusterPoints(TIME, 1024, 6)
            self.columns = None
            self.work = requests(case, seed)
            self.queries = [query(cell, win, avg) for _, _, cell, win, avg in self.work]
            if case["call"] == "batch":
                self.sets = [self.h.polyset(xy, p) for xy, p, _, _, _ in self.work]
            else:
                self.server = self.h.server(slots=2, canvas_mb=16384, max_batch=64)
            return
        dh.setPolygons(*regions(case, seed))
        cons, window = conditions(case)
        dh.setQueryConstraints(cons)
        if window:
            dh.setTimeRange(*window)
        if case["avg"]:
            dh.setAggregation(rj.Avg, VALUE)
        self.h.setDataHandler(dh)
        self.h.setCellSize(case["cell"])
        if case["fresh"]:
            self.h.flags = rj.FLAG_NO_CACHE
        self.fn = FN[case["join"]]
        self.h.upload()
        if case["call"] == "prepared":
            self.plan = self.h.prepare(self.fn)

    def __del__(self):
        for x in [self.server, self.plan] + self.sets:
            if x is not None:
                x.close()


def query(cell, window, avg):
    q = rj.default_query()
    q.function_type = rj.RasterJoinFn
    q.cell_size = cell
    q.time_attrib, q.t_start, q.t_end = TIME, int(window[0]), int(window[1])
    if avg:
        q.aggregation, q.aggr_attrib = rj.Avg, VALUE
    return q


def prepare(case, seed):
    return Program(case, seed)


def run(p):
    call = p.case["call"]
    if call == "batch":
        rs, _, _ = p.h.execute_batch(p.queries, p.sets)
        return answer(rs)
    if call == "served":
        # every request brings its own polygons
        sets, tickets = [], []
        for (xy, pidx, _, _, _), q in zip(p.work, p.queries):
            sets.append(p.h.polyset(xy, pidx))
            tickets.append(p.server.submit(q, sets[-1]))
        rs = [p.server.poll(t)[0] for t in tickets]
        for s in sets:
            s.close()
        return answer(rs)
    r = p.plan.execute() if call == "prepared" else p.h.execute(p.fn)
    out = {"count": r.count, "sum": r.sum, "compat3": r.compat3}
    if r.bounds is not None:
        out["bounds"] = r.bounds
    return out


def answer(results):
    return {"count": np.concatenate([r.count for r in results]), "sum": np.concatenate([r.sum for r in results])}


def work(case):
    """Every row's columns read once, the polygons read once, the results
    written once (rows outside a query's time window are not counted)."""
    n = case["points"]
    if case["call"] == "batch":
        # half the queries average; the windows hold 1e4 rows to all of them
        frac = sum(math.exp(u * math.log(1e4 / n)) for u in ((i + 0.5) / 16 for i in range(16))) / 16
        return {"bytes": min(1.0, frac * case["queries"]) * n * 16.0, "flops": 0.0}
    if case["call"] == "served":
        frac = 0.017 * case["queries"]    # windows of an hour to 30 days, log-uniform
        return {"bytes": min(1.0, frac) * n * 12.0, "flops": 0.0}
    verts = case["npolys"] * (100 if case["polys"] == "cells" else 150)
    return {"bytes": n * (8.0 + 4.0 * (len(columns(case)) - 1)) + 8.0 * verts + 28.0 * case["npolys"], "flops": 0.0}


# ---- exact sums ------------------------------------------------------------
# Counts and bounds are whole numbers; the sums are what 64 bits say.
def rows_kept(cols, cons, window):
    keep = torch.ones(len(cols[LOC]), dtype=torch.bool, device="cuda")
    if window:
        keep &= (cols[TIME] >= int(window[1])) & (cols[TIME] <= int(window[2]))
    for k, op, v in cons:
        keep &= cols[k] > v if op == rj.GT else cols[k] < v
    return keep


def inside(px, py, ring):
    """Even-odd rule in 64 bits: which of the points lie in the ring."""
    x0, y0 = ring[:, 0], ring[:, 1]
    x1, y1 = torch.roll(x0, -1), torch.roll(y0, -1)
    odd = torch.zeros(px.shape, dtype=torch.bool, device="cuda")
    for i in range(len(x0)):
        dy = y1[i] - y0[i]
        cross = (y0[i] > py) != (y1[i] > py)
        at = x0[i] + (py - y0[i]) * (x1[i] - x0[i]) / torch.where(dy == 0, torch.ones_like(dy), dy)
        odd ^= cross & (px < at)
    return odd


def point_sums(xy, v, verts, pidx):
    """Sums over the points inside each polygon (hybrid and index joins)."""
    order = torch.argsort(xy[:, 1])
    x, y, v = xy[order, 0].contiguous(), xy[order, 1].contiguous(), v[order]
    out = np.zeros(len(pidx) - 1)
    rings = torch.from_numpy(verts.astype(np.float64)).cuda()
    for p in range(len(pidx) - 1):
        r = rings[pidx[p]:pidx[p + 1]]
        lo = int(torch.searchsorted(y, r[:, 1].min().float()))
        hi = int(torch.searchsorted(y, r[:, 1].max().float(), right=True))
        near = torch.nonzero((x[lo:hi] >= r[:, 0].min()) & (x[lo:hi] <= r[:, 0].max()))[:, 0] + lo
        if len(near):
            out[p] = v[near][inside(x[near].double(), y[near].double(), r)].sum().item()
    return out


def pixel_sums(xy, v, verts, pidx, cell):
    """Sums over the pixels whose centres lie inside each polygon (raster joins)."""
    lo, hi = verts.min(0).astype(np.float64), verts.max(0).astype(np.float64)
    full = np.ceil((hi - lo) / cell)
    split = np.ceil(full / 8192.0)
    res = (np.ceil(full / split) * split).astype(np.int64)      # whole tiles
    w = torch.from_numpy(res / (hi - lo)).cuda()
    win = torch.round((torch.from_numpy(verts.astype(np.float64) - lo).cuda()) * w * 256.0) / 256.0
    size = (win.max(0).values - win.min(0).values)
    area = sum(float(np.prod(np.ptp(verts[a:b].astype(np.float64), 0) * w.cpu().numpy() + 2))
               for a, b in zip(pidx[:-1], pidx[1:]) if b > a)
    if res[0] * res[1] > 1 << 30 or area > 4e9 or size.max() > 60000:
        return None
    resx, resy = int(res[0]), int(res[1])
    canvas = torch.zeros(resx * resy, dtype=torch.float64, device="cuda")
    for s in range(0, len(xy), 1 << 26):
        at = torch.floor((xy[s:s + (1 << 26)].double() - torch.from_numpy(lo).cuda()) * w).long()
        ok = (at[:, 0] >= 0) & (at[:, 0] < resx) & (at[:, 1] >= 0) & (at[:, 1] < resy)
        canvas.index_add_(0, (at[:, 1] * resx + at[:, 0])[ok], v[s:s + (1 << 26)][ok])
    canvas = canvas.view(resy, resx)
    out = np.zeros(len(pidx) - 1)
    for p in range(len(pidx) - 1):
        r = win[pidx[p]:pidx[p + 1]]
        if len(r) < 3:
            continue
        x0, y0 = int(r[:, 0].min().clamp(0, resx - 1)), int(r[:, 1].min().clamp(0, resy - 1))
        x1, y1 = int(r[:, 0].max().clamp(0, resx - 1)) + 1, int(r[:, 1].max().clamp(0, resy - 1)) + 1
        ay, by = r[:, 1], torch.roll(r[:, 1], -1)
        ax, bx = r[:, 0], torch.roll(r[:, 0], -1)
        cy = torch.arange(y0, y1, device="cuda", dtype=torch.float64) + 0.5
        hit = (ay[None] > cy[:, None]) != (by[None] > cy[:, None])
        row, e = torch.nonzero(hit, as_tuple=True)
        at = ax[e] + (cy[row] - ay[e]) * (bx[e] - ax[e]) / (by[e] - ay[e])
        first = (torch.ceil(at - 0.5).long() - x0).clamp(0, x1 - x0)      # first pixel centre at or right of it
        flips = torch.zeros((y1 - y0, x1 - x0 + 1), dtype=torch.int32, device="cuda")
        flips.view(-1).index_add_(0, row * (x1 - x0 + 1) + first, torch.ones_like(row, dtype=torch.int32))
        odd = (torch.cumsum(flips, 1)[:, :-1] & 1).bool()
        out[p] = canvas[y0:y1, x0:x1][odd].sum().item()
    return out


def exact(case, seed):
    if case["call"] in ("batch", "served"):
        cols = table(case["points"], seed, columns(case))
        sums = []
        for xy, pidx, cell, win, avg in requests(case, seed):
            s = np.zeros(len(pidx) - 1)
            if avg:
                keep = rows_kept(cols, [], (TIME,) + tuple(win))
                s = pixel_sums(cols[LOC][keep], cols[VALUE][keep].double(), xy, pidx, cell)
                if s is None:
                    return None
            sums.append(s)
        return {"count": None, "sum": np.concatenate(sums)}
    verts, pidx = regions(case, seed)
    out = {"count": None, "sum": np.zeros(len(pidx) - 1), "compat3": None}
    if case["join"] == "bounds":
        out["bounds"] = None
    if case["avg"]:
        cols = table(case["points"], seed, columns(case))
        keep = rows_kept(cols, *conditions(case))
        xy, v = cols[LOC][keep], cols[VALUE][keep].double()
        if case["join"] in ("hybrid", "index"):
            out["sum"] = point_sums(xy, v, verts, pidx)
        else:
            out["sum"] = pixel_sums(xy, v, verts, pidx, case["cell"])
            if out["sum"] is None:
                return None
    return out
