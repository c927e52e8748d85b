// rj_poly_kernels.cu -- polygon-side kernels.
//
//  * k_transform_vertices : world -> per-tile window coordinates (float and
//    1/256-pixel fixed point), the vertex stage of polygon.vert:9-13.
//  * k_poly_info          : per (tile, polygon) the pixels and rows it can reach.
//  * k_poly_label         : a flat map of polygon labels by edge-function
//    coverage of pixel centres (the passes over point canvases are in
//    rj_band_kernels.cu).
//  * grid index build     : index-size.glsl + create-index.glsl as a CSR grid.
//  * hybrid border mask   : outline pass of HybridJoin::drawOutline
//    (HybridJoin.cpp:197-268) as a conservative supercover + dilation.
#include <climits>
#include <cstdio>
#include <map>
#include <mutex>

#include "rj_bands.cuh"
#include "rj_launch.h"

namespace rj {

thread_local int g_kernel_launches = 0;

cudaError_t allow_smem(const void* kernel, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> allowed;   // (device, kernel)
    // What this thread last saw allowed (one slot a kernel); most launches need no
    // more.  With the lock and the map every time a count of 20,000 points took
    // 88.1 us instead of 86.8.
    struct Seen {
        const void* kernel;
        int dev;
        size_t bytes;
    };
    static thread_local Seen seen[64];
    if (bytes <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    Seen& s = seen[(reinterpret_cast<uintptr_t>(kernel) >> 4) % 64];
    if (s.kernel == kernel && s.dev == dev && bytes <= s.bytes) return cudaSuccess;
    std::lock_guard<std::mutex> lock(mu);
    size_t& now = allowed[{dev, kernel}];
    if (bytes > now) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        now = bytes;
    }
    s = {kernel, dev, now};
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// tile column and row transforms: (sx, tx, hx, -) and (sy, ty, hy, -)
template <class COL, class ROW>
__device__ __forceinline__ void transform_vertices(const float2* __restrict__ verts, int V, COL&& col, ROW&& row, int splitx,
                                                   int T, int2* __restrict__ wv, float2* __restrict__ wf) {
    size_t total = (size_t)T * V;
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < total; g += (size_t)gridDim.x * blockDim.x) {
        int t = (int)(g / V);
        int v = (int)(g - (size_t)t * V);
        const float4 cxf = col(t % splitx), ryf = row(t / splitx);
        float2 p = __ldg(verts + v);
        float wx = win_coord(p.x, cxf.x, cxf.y, cxf.z);
        float wy = win_coord(p.y, ryf.x, ryf.y, ryf.z);
        wv[g] = make_int2(snap_win(wx), snap_win(wy));
        if (wf) wf[g] = make_float2(wx, wy);
    }
}

__global__ void k_transform_vertices(const float2* verts, int V, const float4* __restrict__ colxf,
                                     const float4* __restrict__ rowxf, int splitx, int T, int2* wv, float2* wf) {
    transform_vertices(verts, V, [&](int c) { return __ldg(colxf + c); }, [&](int r) { return __ldg(rowxf + r); }, splitx, T,
                       wv, wf);
}

// the transforms as arguments, also written where the later passes read them
__global__ void k_transform_vertices_xf(const float2* verts, int V, __grid_constant__ const XfArgs col,
                                        __grid_constant__ const XfArgs row, int splitx, int T, int2* wv, float2* wf,
                                        float4* dcol, float4* drow) {
    if (blockIdx.x == 0 && threadIdx.x < kXfArgs) {
        if ((int)threadIdx.x < splitx) dcol[threadIdx.x] = col.v[threadIdx.x];
        if ((int)threadIdx.x < T / splitx) drow[threadIdx.x] = row.v[threadIdx.x];
    }
    transform_vertices(verts, V, [&](int c) { return col.v[c]; }, [&](int r) { return row.v[r]; }, splitx, T, wv, wf);
}

// ---------------------------------------------------------------------------
constexpr int kPolyWarps = 8;
constexpr int kBandCap = 256;      // staged edges per warp
constexpr int kCrossCap = 512;     // crossings per row per warp (sorted into spans)
// dynamic shared memory of k_poly_label: per warp the staged edges and one
// row's crossings
constexpr size_t kPolySmem = (size_t)kPolyWarps * (kBandCap * sizeof(int4) + kCrossCap * sizeof(int));

// Ascending sort of buf[0, m) by one warp (bitonic network in shared memory,
// m padded to a power of two with INT_MAX).
__device__ __forceinline__ void warp_sort_ints(int* buf, int m, int lane) {
    int mp = 2;
    while (mp < m) mp <<= 1;
    for (int i = m + lane; i < mp; i += 32) buf[i] = INT_MAX;
    __syncwarp();
    for (int k = 2; k <= mp; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < mp; i += 32) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const int x = buf[i], y = buf[ixj];
                    const bool up = (i & k) == 0;
                    if ((x > y) == up) {
                        buf[i] = y;
                        buf[ixj] = x;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// Per (tile, polygon): pixel column range that can be covered, rows to visit
// and rows whose centre line the polygon can cross; number of row bands.
template <int MODE>
__global__ void k_poly_info(PolyPassArgs a) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int TP = a.T * a.P;
    for (int item = wid; item < TP; item += nw) {
        const int t = item / a.P, p = item - t * a.P;
        const int v0 = __ldg(a.pindex + p);
        const int n = __ldg(a.pindex + p + 1) - v0;
        const int2* pv = a.wv + (size_t)t * a.V + v0;
        int xmin = INT_MAX, xmax = INT_MIN, ymin = INT_MAX, ymax = INT_MIN;
        for (int k = lane; k < n; k += 32) {
            int2 q = pv[k];
            xmin = min(xmin, q.x); xmax = max(xmax, q.x);
            ymin = min(ymin, q.y); ymax = max(ymax, q.y);
        }
        xmin = warp_min(xmin); xmax = warp_max(xmax);
        ymin = warp_min(ymin); ymax = warp_max(ymax);
        if (lane != 0) continue;
        int nbands = 0;
        int4 ia = make_int4(0, -1, 0, -1);
        int2 ib = make_int2(0, -1);
        if (n >= 2) {
            // rows whose centre can be crossed: ymin < Cy <= ymax
            int j_lo = (int)floordiv64((int64_t)ymin - kSub / 2, kSub) + 1;
            int j_hi = (int)floordiv64((int64_t)ymax - kSub / 2, kSub);
            // pixels that can be inside: ceil((xmin-128)/256) .. ceil((xmax-128)/256)-1
            int i_lo = (int)floordiv64((int64_t)xmin - kSub / 2 + kSub - 1, kSub);
            int i_hi = (int)floordiv64((int64_t)xmax - kSub / 2 + kSub - 1, kSub) - 1;
            int r_lo = j_lo, r_hi = j_hi;
            const bool outline = MODE == MODE_BOUNDS || (MODE == MODE_TIER_CLASSIFY && a.outline_rows);
            if (outline) {
                // rows whose pixel rectangle an edge may touch
                r_lo = min(r_lo, (int)floordiv64((int64_t)ymin, kSub) - 1);
                r_hi = max(r_hi, (int)floordiv64((int64_t)ymax, kSub) + 1);
            }
            r_lo = max(r_lo, 0);
            r_hi = min(r_hi, a.resy - 1);
            if (MODE >= MODE_TIER_CLASSIFY) r_lo &= ~15;   // bands on block rows
            i_lo = max(i_lo, 0);
            i_hi = min(i_hi, a.resx - 1);
            if (r_lo <= r_hi && (outline || i_lo <= i_hi)) {
                nbands = (r_hi - r_lo + kBand) / kBand;
                ia = make_int4(i_lo, i_hi, r_lo, r_hi);
                ib = make_int2(j_lo, j_hi);
            }
        }
        a.info_a[item] = ia;
        a.info_b[item] = ib;
        a.nbands[item] = nbands;
    }
}

// Flat label map.  One warp per (tile, polygon, band of kBand rows): the band's
// edges are staged in shared memory, each row's centre-line crossings are
// computed exactly, and every pixel of the row is inside iff an odd number of
// crossings lies to its right.
__global__ void __launch_bounds__(kPolyWarps * 32)
k_poly_label(PolyPassArgs a) {
    extern __shared__ int4 s_poly[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    const int TP = a.T * a.P;
    BandItems work(a.band_start, TP, a.work_ctr, kPolyWarps, warp, lane);
    int4* my_edge = s_poly + (size_t)warp * kBandCap;
    int* my_cross = reinterpret_cast<int*>(s_poly + (size_t)kPolyWarps * kBandCap) + (size_t)warp * kCrossCap;

    for (;;) {
        const int item = work.take(a.band_start, TP, a.work_ctr, lane);
        if (item < 0) break;
        const int tp = work.tp;
        const int t = tp / a.P, p = tp - t * a.P;
        const int band = item - work.tp_first;
        const int4 ia = a.info_a[tp];
        const int2 ib = a.info_b[tp];
        const int i_lo = ia.x, i_hi = ia.y, j_lo = ib.x, j_hi = ib.y;
        const int jb = ia.z + band * kBand;
        const int je = min(jb + kBand - 1, ia.w);
        const int v0 = __ldg(a.pindex + p);
        const int n = __ldg(a.pindex + p + 1) - v0;
        const int2* pv = a.wv + (size_t)t * a.V + v0;
        const size_t tile_off = (size_t)t * a.resx * a.resy;
        unsigned long long covered = 0;

        // fixed-point y window of the band (one pixel of margin each side)
        const int64_t band_lo = (int64_t)jb * kSub - kSub;
        const int64_t band_hi = (int64_t)(je + 1) * kSub + kSub;
        const int nb = stage_edges(pv, n, band_lo, band_hi, lane, [&](int pos, int, const int4& e) {
            if (pos < kBandCap) my_edge[pos] = e;
        });
        const bool overflow = nb > kBandCap;
        __syncwarp();

        for (int j = max(jb, j_lo); j <= min(je, j_hi); ++j) {
            const int32_t cy = j * kSub + kSub / 2;
            // crossings of this row's centre line: from the staged edges, or
            // from all edges of the polygon when the band held too many
            int m = 0;
            const int ne = overflow ? n : nb;
            for (int e0 = 0; e0 < ne; e0 += 32) {
                const int e = e0 + lane;
                bool c = false;
                int L = 0;
                if (e < ne) {
                    int4 q;
                    if (!overflow) {
                        q = my_edge[e];
                    } else {
                        const int2 A = pv[e];
                        const int2 B = pv[(e + 1 == n) ? 0 : e + 1];
                        q = make_int4(A.x, A.y, B.x, B.y);
                    }
                    if (cross_row(q.y, q.w, cy)) { c = true; L = cross_L(q.x, q.y, q.z, q.w, cy); }
                }
                const unsigned bm = __ballot_sync(FULL, c);
                const int pos = m + __popc(bm & ((1u << lane) - 1u));
                if (c && pos < kCrossCap) my_cross[pos] = L;
                m += __popc(bm);
            }
            __syncwarp();
            // pixel i is covered when an odd number of crossings lie at or
            // left of it: with the crossings sorted, [c0, c1), [c2, c3), ...
            // (overlaps are detected by counting, see k_label_finish)
            uint16_t* row = a.label + tile_off + (size_t)j * a.resx;
            if (m <= kCrossCap) {
                warp_sort_ints(my_cross, m, lane);
                for (int s2 = 0; s2 + 1 < m; s2 += 2) {
                    const int L = max(my_cross[s2], i_lo), R = min(my_cross[s2 + 1], i_hi + 1);
                    for (int i = L + lane; i < R; i += 32) {
                        row[i] = (uint16_t)p;
                        ++covered;
                    }
                }
            } else {
                for (int i = i_lo + lane; i <= i_hi; i += 32) {
                    bool inside = false;
                    for (int k = 0; k < n; ++k) {
                        int2 A = pv[k];
                        int2 B = pv[(k + 1 == n) ? 0 : k + 1];
                        if (cross_row(A.y, B.y, cy)) inside ^= (i < cross_L(A.x, A.y, B.x, B.y, cy));
                    }
                    if (inside) {
                        row[i] = (uint16_t)p;
                        ++covered;
                    }
                }
            }
            __syncwarp();
        }
        covered = warp_sum_u64(covered);
        if (lane == 0 && covered) atomicAdd(a.covered, covered);
    }
}

// ---------------------------------------------------------------------------
// Grid index (GLFunction::createPolyIndex GLFunction.cpp:65-156).  One warp
// per polygon: MBR in fp32, cell range as index-size.glsl:50-68 with the
// upper bound clamped to res (default) or res-1 (compat, create-index.glsl:56-61).
__device__ __forceinline__ void poly_cells(const float2* __restrict__ verts, const int* __restrict__ pindex,
                                           const GridArgs& g, int p, int lane,
                                           int& stx, int& sty, int& enx, int& eny) {
    const int v0 = __ldg(pindex + p), n = __ldg(pindex + p + 1) - v0;
    float lbx = INFINITY, lby = INFINITY, rtx = -INFINITY, rty = -INFINITY;
    for (int k = lane; k < n; k += 32) {
        float2 q = __ldg(verts + v0 + k);
        lbx = fminf(lbx, q.x); rtx = fmaxf(rtx, q.x);
        lby = fminf(lby, q.y); rty = fmaxf(rty, q.y);
    }
    lbx = warp_minf(lbx); rtx = warp_maxf(rtx);
    lby = warp_minf(lby); rty = warp_maxf(rty);
    stx = __float2int_rz(__fdiv_rn(__fsub_rn(lbx, g.lbx), g.csx));
    sty = __float2int_rz(__fdiv_rn(__fsub_rn(lby, g.lby), g.csy));
    enx = __float2int_rz(__fdiv_rn(__fsub_rn(rtx, g.lbx), g.csx)) + 1;
    eny = __float2int_rz(__fdiv_rn(__fsub_rn(rty, g.lby), g.csy)) + 1;
    const int cap = g.compat_clamp ? g.res - 1 : g.res;
    if (enx >= cap) enx = cap;
    if (eny >= cap) eny = cap;
    if (stx < 0) stx = 0;
    if (sty < 0) sty = 0;
    if (n == 0) { enx = stx; eny = sty; }
}

__global__ void k_grid_count(GridArgs g) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = wid; p < g.P; p += nw) {
        int stx, sty, enx, eny;
        poly_cells(g.verts, g.pindex, g, p, lane, stx, sty, enx, eny);
        const int w = enx - stx, h = eny - sty;
        if (w <= 0 || h <= 0) continue;
        for (int c = lane; c < w * h; c += 32) {
            int x = stx + c % w, y = sty + c / w;
            atomicAdd(g.cell_count + (size_t)y * g.res + x, 1);
        }
    }
}

__global__ void k_grid_fill(GridArgs g) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = wid; p < g.P; p += nw) {
        int stx, sty, enx, eny;
        poly_cells(g.verts, g.pindex, g, p, lane, stx, sty, enx, eny);
        const int w = enx - stx, h = eny - sty;
        if (w <= 0 || h <= 0) continue;
        for (int c = lane; c < w * h; c += 32) {
            int x = stx + c % w, y = sty + c / w;
            size_t cell = (size_t)y * g.res + x;
            int pos = g.cell_start[cell] + atomicAdd(g.cursor + cell, 1);
            g.entries[pos] = p;
            if (g.pair_cell) g.pair_cell[pos] = (int)cell;
        }
    }
}

// Deterministic order inside each cell: ascending polygon id.
__global__ void k_grid_sort(const int* __restrict__ cell_start, int* __restrict__ entries, int ncells) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x) {
        int s = cell_start[c], e = cell_start[c + 1];
        for (int i = s + 1; i < e; ++i) {
            int v = entries[i], j = i - 1;
            while (j >= s && entries[j] > v) { entries[j + 1] = entries[j]; --j; }
            entries[j + 1] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Classified grid.  For the pair (cell c, polygon p) let R be the cell grown
// by `margin` (>= the fp32 error of the crossing test, of the point-to-cell
// assignment and of the relative coordinates used here).  If no edge of p
// meets R, every point assigned to c has the same crossing-number result as
// the cell centre: the pair is FULL or OUT.  Otherwise only edges whose
// y-extent meets R's rows can toggle a point of c; of those, edges entirely
// left of R never toggle and edges entirely right of R toggle exactly when
// they straddle the point's y.
// Level 1 classifies the candidate pairs on the coarse (query) grid; FULL and
// OUT results hold for every fine cell inside, EDGE pairs are refined into
// their scale x scale fine cells and classified again (level 2), keeping the
// edge lists of the fine EDGE pairs.
struct CellRect {
    float cx, cy;      // centre
    float hw, hh;      // half extents grown by the margin
};

__device__ __forceinline__ int pair_poly(const ClsArgs& a, int k) {
    int lo = 0, hi = a.P - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(a.pair_off + mid) <= k) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// rectangle of fine cells [gx, gx+n) x [gy, gy+n) of the fine grid.  The edges
// of a pair are counted by one kernel and written by another: every rounding is
// spelled out, so that both see the same rectangle.
__device__ __forceinline__ CellRect cells_rect(const ClsArgs& a, int gx, int gy, int n) {
    // cell 0 also receives points with (p - lb)/cs in (-1, 0): int() truncates
    const float x0 = __fmaf_rn(gx == 0 ? -1.0f : (float)gx, a.csx, a.lbx), x1 = __fmaf_rn((float)(gx + n), a.csx, a.lbx);
    const float y0 = __fmaf_rn(gy == 0 ? -1.0f : (float)gy, a.csy, a.lby), y1 = __fmaf_rn((float)(gy + n), a.csy, a.lby);
    CellRect r;
    r.cx = __fmul_rn(0.5f, __fadd_rn(x0, x1));
    r.cy = __fmul_rn(0.5f, __fadd_rn(y0, y1));
    r.hw = __fadd_rn(__fmul_rn(0.5f, __fsub_rn(x1, x0)), a.margin);
    r.hh = __fadd_rn(__fmul_rn(0.5f, __fsub_rn(y1, y0)), a.margin);
    return r;
}

// Does the segment a-b meet the box [-hw,hw] x [-hh,hh]?  (Liang-Barsky)
__device__ __forceinline__ bool seg_meets_box(float ax, float ay, float bx, float by, float hw, float hh) {
    if (fmaxf(ax, bx) < -hw || fminf(ax, bx) > hw || fmaxf(ay, by) < -hh || fminf(ay, by) > hh) return false;
    float t0 = 0.0f, t1 = 1.0f;
    const float dx = bx - ax, dy = by - ay;
    const float p[4] = {-dx, dx, -dy, dy};
    const float q[4] = {ax + hw, hw - ax, ay + hh, hh - ay};
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (p[i] == 0.0f) {
            if (q[i] < 0.0f) return false;
        } else {
            float r = q[i] / p[i];
            if (p[i] < 0.0f) t0 = fmaxf(t0, r);
            else t1 = fminf(t1, r);
            if (t0 > t1) return false;
        }
    }
    return true;
}

// per edge of the pair: bit0 meets R, bit1 kept (may toggle), bit2 straddle-only
__device__ __forceinline__ int edge_class(const CellRect& r, float2 vi, float2 vj) {
    const float ax = __fsub_rn(vi.x, r.cx), ay = __fsub_rn(vi.y, r.cy);
    const float bx = __fsub_rn(vj.x, r.cx), by = __fsub_rn(vj.y, r.cy);
    int c = seg_meets_box(ax, ay, bx, by, r.hw, r.hh) ? 1 : 0;
    const bool band = !(fmaxf(ay, by) < -r.hh || fminf(ay, by) > r.hh) && !(fmaxf(ax, bx) < -r.hw);
    if (band) {
        c |= 2;
        if (fminf(ax, bx) > r.hw) c |= 4;
    }
    return c;
}

// The polygon's edges, 32 at a time in order, as f(end, start, live) by
// the whole warp; groups with no edge in the rectangle's rows, which neither
// meet it nor toggle anything, are passed over.  An outline is local, so few
// groups are left, and the loads of four are in flight at a time.
template <class F>
__device__ __forceinline__ void for_near_edges(const float2* __restrict__ v, int nv, const CellRect& r, int lane, F&& f) {
    for (int e0 = 0; e0 < nv; e0 += 128) {
        float2 vi[4], vj[4];
        #pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + 32 * u + lane;
            const bool live = e < nv;
            vi[u] = live ? __ldg(v + e) : make_float2(0.f, 0.f);
            vj[u] = live ? __ldg(v + (e == 0 ? nv - 1 : e - 1)) : make_float2(0.f, 0.f);
        }
        #pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool live = e0 + 32 * u + lane < nv;
            const float ay = __fsub_rn(vi[u].y, r.cy), by = __fsub_rn(vj[u].y, r.cy);
            if (__any_sync(0xffffffffu, live && !(fmaxf(ay, by) < -r.hh || fminf(ay, by) > r.hh)))
                f(vi[u], vj[u], live);
        }
    }
}

// What the edges say about one (cell, polygon) pair.
struct PairEdges {
    int meets = 0, nr = 0, nf = 0;
    bool inside = false;
};

__device__ __forceinline__ PairEdges pair_edges_warp(const float2* __restrict__ v, int nv, const CellRect& r, int lane) {
    const unsigned FULL = 0xffffffffu;
    PairEdges t;
    for_near_edges(v, nv, r, lane, [&](float2 vi, float2 vj, bool live) {
        int c = 0;
        bool tog = false;
        if (live) {
            c = edge_class(r, vi, vj);
            tog = edge_toggles(vi.x, vi.y, vj.x, vj.y, r.cx, r.cy);
        }
        t.meets |= __any_sync(FULL, c & 1);
        t.nr += __popc(__ballot_sync(FULL, (c & 6) == 6));
        t.nf += __popc(__ballot_sync(FULL, (c & 6) == 2));
        t.inside ^= (__popc(__ballot_sync(FULL, tog)) & 1) != 0;
    });
    return t;
}

// Levels 1 and 3, a pair per lane: neighbouring pairs mostly share their polygon,
// so each of its edges is one broadcast load and a few comparisons for 32 cells.
// Edges left of the cell's rectangle say nothing, edges right of it only
// whether they straddle its middle; the others are marked, and the lanes then
// work off their own marks together.  With a warp per pair (the edges over the
// lanes) a pair is one load latency after another, whatever its edges are:
// 65,000 cells of 260 polygons with 100 vertices, 120,000 pairs, took 89 us and
// 19 more for level 2; 38 us now for both.  Polygons of more than kLaneEdges
// vertices are still walked by the warp, pair by pair: a lane alone would be at
// it for too long.
constexpr int kLaneEdges = 512;

__global__ void __launch_bounds__(128, 6) k_cls_pairs(ClsArgs a) {
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    for (int k0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) & ~31u); k0 < a.npairs; k0 += (int)(gridDim.x * blockDim.x)) {
        const int k = k0 + lane;
        const bool valid = k < a.npairs;
        int p = -1, gx = 0, gy = 0;
        const int n = a.scale;
        if (valid) {
            p = pair_poly(a, k);
            const int4 r = __ldg(a.prange + p);
            const int w = r.y - r.x, l = k - __ldg(a.pair_off + p);
            gx = (r.x + l % w) * n;
            gy = (r.z + l / w) * n;
        }
        const CellRect r = cells_rect(a, gx, gy, n);
        PairEdges res;
        for (unsigned todo = __ballot_sync(FULL, valid); todo;) {
            const int pl = __shfl_sync(FULL, p, __ffs(todo) - 1);
            const bool mine = p == pl;
            const unsigned group = __ballot_sync(FULL, mine);
            todo &= ~group;
            const int v0 = __ldg(a.pindex + pl), nv = __ldg(a.pindex + pl + 1) - v0;
            const float2* v = a.verts + v0;
            if (nv <= kLaneEdges) {
                float2 vj = nv ? __ldg(v + nv - 1) : make_float2(0.f, 0.f);
                for (int e0 = 0; e0 < nv; e0 += 32) {
                    unsigned marks = 0u;
                    #pragma unroll 1
                    for (int e1 = 0; e1 < 32 && e0 + e1 < nv; e1 += 8) {
                        float2 vi[8];
                        #pragma unroll
                        for (int u = 0; u < 8; ++u) vi[u] = __ldg(v + min(e0 + e1 + u, nv - 1));
                        #pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float ax = __fsub_rn(vi[u].x, r.cx), ay = __fsub_rn(vi[u].y, r.cy);
                            const float bx = __fsub_rn(vj.x, r.cx), by = __fsub_rn(vj.y, r.cy);
                            if (mine && e0 + e1 + u < nv && !(fmaxf(ay, by) < -r.hh || fminf(ay, by) > r.hh) &&
                                !(ax < -r.hw && bx < -r.hw)) {
                                if (ax > r.hw && bx > r.hw) {
                                    ++res.nr;
                                    res.inside ^= (vi[u].y > r.cy) != (vj.y > r.cy);
                                } else {
                                    marks |= 1u << (e1 + u);
                                }
                            }
                            vj = vi[u];
                        }
                    }
                    while (__any_sync(FULL, marks != 0u)) {
                        if (marks) {
                            const int e = e0 + __ffs(marks) - 1;
                            marks &= marks - 1;
                            const float2 vi = __ldg(v + e), vp = __ldg(v + (e == 0 ? nv - 1 : e - 1));
                            const int c = edge_class(r, vi, vp);
                            res.meets |= c & 1;
                            res.nr += (c & 6) == 6;
                            res.nf += (c & 6) == 2;
                            res.inside ^= edge_toggles(vi.x, vi.y, vp.x, vp.y, r.cx, r.cy);
                        }
                    }
                }
            } else {
                for (unsigned g = group; g; g &= g - 1) {
                    const int who = __ffs(g) - 1;
                    const CellRect rr{__shfl_sync(FULL, r.cx, who), __shfl_sync(FULL, r.cy, who),
                                      __shfl_sync(FULL, r.hw, who), __shfl_sync(FULL, r.hh, who)};
                    const PairEdges t = pair_edges_warp(v, nv, rr, lane);
                    if (lane == who) res = t;
                }
            }
        }
        const int kind = res.meets ? 0 : (res.inside ? -1 : -2);
        const int cell = gy * a.res + gx;
        if (a.level == 3) {   // one fine cell per coarse cell: this is level 2 as well
            if (valid) {
                a.info[k] = (kind == 0) ? make_int4(p, res.nr, res.nf, cell) : make_int4(p, kind, 0, cell);
                a.ecount[k] = (kind == 0) ? res.nr + res.nf : 0;
                if (kind != -2) atomicAdd(a.cell_kept + cell, 1);
            }
            continue;
        }
        if (valid) a.info[k] = make_int4(p, kind, 0, cell);
        // the fine cells of full and of edge pairs, pair by pair
        for (unsigned m = __ballot_sync(FULL, valid && kind == -1); m; m &= m - 1) {
            const int x = __shfl_sync(FULL, gx, __ffs(m) - 1), y = __shfl_sync(FULL, gy, __ffs(m) - 1);
            for (int s = lane; s < n * n; s += 32) atomicAdd(a.cell_kept + (y + s / n) * a.res + x + s % n, 1);
        }
        unsigned m = __ballot_sync(FULL, valid && kind == 0);
        int base = 0;
        if (m && lane == 0) base = atomicAdd(a.plist_n, __popc(m) * n * n);
        base = __shfl_sync(FULL, base, 0);
        for (; m; m &= m - 1) {
            const int who = __ffs(m) - 1;
            const int q = __shfl_sync(FULL, p, who), x = __shfl_sync(FULL, gx, who), y = __shfl_sync(FULL, gy, who);
            for (int s = lane; s < n * n; s += 32) a.plist[base + s] = make_int2(q, (y + s / n) * a.res + x + s % n);
            base += n * n;
        }
    }
}

// A pair per warp: level 2, whose list mixes polygons, and the other levels when
// there are too few pairs to give every warp 32 (launch_cls_classify).
__global__ void k_cls_classify(ClsArgs a) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int npairs = a.level == 2 ? *a.plist_n : a.npairs;
    const int n = a.level == 1 ? a.scale : 1;
    for (int k = wid; k < npairs; k += nw) {
        int p, gx, gy;
        if (a.level == 2) {
            const int2 q = a.plist[k];
            p = q.x;
            gx = q.y % a.res;
            gy = q.y / a.res;
        } else {
            p = pair_poly(a, k);
            const int4 r = __ldg(a.prange + p);
            const int w = r.y - r.x, l = k - __ldg(a.pair_off + p);
            gx = (r.x + l % w) * n;
            gy = (r.z + l / w) * n;
        }
        const int v0 = __ldg(a.pindex + p), nv = __ldg(a.pindex + p + 1) - v0, cell = gy * a.res + gx;
        const PairEdges t = pair_edges_warp(a.verts + v0, nv, cells_rect(a, gx, gy, n), lane);
        const int kind = t.meets ? 0 : (t.inside ? -1 : -2);
        if (a.level == 1) {
            if (lane == 0) a.info[k] = make_int4(p, kind, 0, cell);
            int base = 0;
            if (kind == 0 && lane == 0) base = atomicAdd(a.plist_n, n * n);
            base = __shfl_sync(0xffffffffu, base, 0);
            for (int s = lane; s < n * n; s += 32) {
                const int c = (gy + s / n) * a.res + gx + s % n;
                if (kind == -1) atomicAdd(a.cell_kept + c, 1);
                else if (kind == 0) a.plist[base + s] = make_int2(p, c);
            }
        } else if (lane == 0) {
            a.info[k] = (kind == 0) ? make_int4(p, t.nr, t.nf, cell) : make_int4(p, kind, 0, cell);
            a.ecount[k] = (kind == 0) ? t.nr + t.nf : 0;
            if (kind != -2) atomicAdd(a.cell_kept + cell, 1);
        }
    }
}

// Kept pairs into the cell-major list (order inside a cell is immaterial).
// Level 1: FULL coarse pairs expand to their fine cells.  Level 2: kept pairs.
__global__ void k_cls_emit(ClsArgs a) {
    const int npairs = a.level == 2 ? *a.plist_n : a.npairs;
    const int nn = a.scale * a.scale;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < npairs; k += gridDim.x * blockDim.x) {
        int4 in = a.info[k];
        if (a.level == 1) {
            if (in.y != -1) continue;
            const int gx = in.w % a.res, gy = in.w / a.res;
            for (int s = 0; s < nn; ++s) {
                const int cell = (gy + s / a.scale) * a.res + gx + s % a.scale;
                const int pos = a.cell_start[cell] + atomicAdd(a.cursor + cell, 1);
                a.entries[pos] = make_int4(in.x, -1, 0, 0);
            }
        } else {
            if (in.y == -2) continue;
            const int cell = in.w;
            const int pos = a.cell_start[cell] + atomicAdd(a.cursor + cell, 1);
            in.w = (in.y >= 0) ? a.eoff[k] : 0;
            if (in.y < 0) in.z = 0;
            a.entries[pos] = in;
        }
    }
}

// Level 2: edge lists of fine EDGE pairs (straddle-only edges first).
__global__ void k_cls_fill_edges(ClsArgs a) {
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const unsigned FULL = 0xffffffffu;
    const int npairs = a.level == 2 ? *a.plist_n : a.npairs;
    for (int k = wid; k < npairs; k += nw) {
        if (a.ecount[k] == 0) continue;
        const int4 in = a.info[k];
        const int p = in.x, cell = in.w, nr = in.y;
        const int v0 = __ldg(a.pindex + p), nv = __ldg(a.pindex + p + 1) - v0;
        const CellRect r = cells_rect(a, cell % a.res, cell / a.res, 1);
        float4* out = a.edges + a.eoff[k];
        int wr = 0, wf = nr;
        for_near_edges(a.verts + v0, nv, r, lane, [&](float2 vi, float2 vj, bool live) {
            const int c = live ? edge_class(r, vi, vj) : 0;
            const bool is_r = (c & 6) == 6, is_f = (c & 6) == 2;
            const unsigned mr = __ballot_sync(FULL, is_r), mf = __ballot_sync(FULL, is_f);
            const unsigned below = (1u << lane) - 1u;
            if (is_r) out[wr + __popc(mr & below)] = make_float4(vi.x, vi.y, vj.x, vj.y);
            if (is_f) out[wf + __popc(mf & below)] = make_float4(vi.x, vi.y, vj.x, vj.y);
            wr += __popc(mr);
            wf += __popc(mf);
        });
    }
}

// Count labelled pixels (a polygon set overlaps iff fewer pixels carry a
// label than polygon coverages were written) and fuse the dilated border mask
// of the hybrid canvas into the label map.
__global__ void k_label_finish(uint16_t* __restrict__ label, const uint32_t* __restrict__ mask, int resx, int resy,
                               int ntiles, int words, unsigned long long* __restrict__ nonempty) {
    // A warp takes a row, eight pixels (16 bytes) per lane where the rows are
    // aligned: the map was just written and comes from L2.  On 4096 x 4096
    // pixels 50 us with two-byte loads, a run of 32 pixels per thread; 14 us now.
    const int lane = threadIdx.x & 31;
    const size_t rows = (size_t)resy * ntiles;
    const bool wide = (resx & 7) == 0;
    unsigned long long cnt = 0;
    for (size_t row = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5; row < rows;
         row += ((size_t)gridDim.x * blockDim.x) >> 5) {
        uint16_t* l = label + row * resx;
        const uint32_t* mrow = mask ? mask + (row % resy) * words : nullptr;
        if (wide) {
            uint4* l8 = reinterpret_cast<uint4*>(l);
            #pragma unroll 4
            for (int g = lane; g < resx >> 3; g += 32) {
                uint4 v = l8[g];
                const uint32_t m = mrow ? __ldg(mrow + (g >> 2)) >> ((g & 3) * 8) & 0xFFu : 0u;
                cnt += 8 - ((__popc(__vcmpeq2(v.x, kEmptyLabel * 0x10001u)) + __popc(__vcmpeq2(v.y, kEmptyLabel * 0x10001u)) +
                             __popc(__vcmpeq2(v.z, kEmptyLabel * 0x10001u)) + __popc(__vcmpeq2(v.w, kEmptyLabel * 0x10001u))) >> 4);
                if (m) {
                    const auto mark = [&](uint32_t w, int k) {
                        const uint32_t sel = ((m >> k) & 1u ? 0xFFFFu : 0u) | ((m >> k) & 2u ? 0xFFFF0000u : 0u);
                        return (w & ~sel) | (kBorderLabel * 0x10001u & sel);
                    };
                    l8[g] = make_uint4(mark(v.x, 0), mark(v.y, 2), mark(v.z, 4), mark(v.w, 6));
                }
            }
        } else {
            for (int i = lane; i < resx; i += 32) {
                cnt += l[i] != kEmptyLabel;
                if (mrow && (__ldg(mrow + (i >> 5)) >> (i & 31)) & 1u) l[i] = kBorderLabel;
            }
        }
    }
    cnt = warp_sum_u64(cnt);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(nonempty, cnt);
}

// Per classified cell: the polygon id when the cell lies inside exactly one
// polygon and needs no test, else kCodeEmpty / kCodeList.
__global__ void k_cls_codes(const int* __restrict__ cell_start, const int4* __restrict__ entries,
                            uint32_t* __restrict__ code, int ncells) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x) {
        const int s = cell_start[c], e = cell_start[c + 1];
        uint32_t v;
        if (e == s) v = kCodeEmpty;
        else if (e == s + 1 && entries[s].y == -1) v = (uint32_t)entries[s].x;
        else v = kCodeList;
        code[c] = v;
    }
}

// ---------------------------------------------------------------------------
// Exclusive scan of int counts (n <= 16M) into out[0..n]; out[n] = total.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ int block_exclusive_scan(int v, int* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < (blockDim.x >> 5)) ? s_warp[lane] : 0;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    int base = warp ? s_warp[warp - 1] : 0;
    int r = base + x - v;
    __syncthreads();
    return r;
}

__global__ void k_scan_tiles(const int* in, int* out, int n, int* __restrict__ tile_sums) {
    __shared__ int s_warp[32];
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    int v[kScanItems];
    int local = 0;
    #pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        size_t i = base + k;
        v[k] = (i < (size_t)n) ? in[i] : 0;
        local += v[k];
    }
    int ex = block_exclusive_scan(local, s_warp);
    #pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        size_t i = base + k;
        if (i < (size_t)n) out[i] = ex;
        ex += v[k];
    }
    if (threadIdx.x == blockDim.x - 1) tile_sums[blockIdx.x] = ex;
}

__global__ void k_scan_sums(int* __restrict__ tile_sums, int ntiles, int* __restrict__ total_out) {
    // single block: exclusive scan of tile sums (ntiles <= 4096)
    __shared__ int s_warp[32];
    int v[kScanItems];
    int local = 0;
    #pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int i = threadIdx.x * kScanItems + k;
        v[k] = (i < ntiles) ? tile_sums[i] : 0;
        local += v[k];
    }
    int ex = block_exclusive_scan(local, s_warp);
    #pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int i = threadIdx.x * kScanItems + k;
        if (i < ntiles) tile_sums[i] = ex;
        ex += v[k];
    }
    if (threadIdx.x == blockDim.x - 1) *total_out = ex;
}

// Short arrays: one block, tile after tile.
__global__ void __launch_bounds__(kScanThreads) k_scan_small(const int* in, int* out, int n) {
    __shared__ int s_warp[32];
    __shared__ int s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (int base = 0; base < n; base += kScanTile) {
        const int i0 = base + (int)threadIdx.x * kScanItems;
        int v[kScanItems], local = 0;
        #pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = i0 + k < n ? in[i0 + k] : 0;
            local += v[k];
        }
        int ex = s_carry + block_exclusive_scan(local, s_warp);
        #pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (i0 + k < n) out[i0 + k] = ex;
            ex += v[k];
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) s_carry = ex;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[n] = s_carry;
}

__global__ void k_scan_add(int* __restrict__ out, int n, const int* __restrict__ tile_sums) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (size_t)n) out[i] += tile_sums[i / kScanTile];
}

// ---------------------------------------------------------------------------
// Hybrid border mask.  Window coordinates follow hybrid.glsl rasterize()
// without the range test; every pixel whose rectangle, grown by `margin`
// pixels, meets an edge is marked (a conservative superset of the outline
// fragments of line-simple.frag).
__device__ __forceinline__ void hyb_win(const HybXf& h, float x, float y, float& u, float& v) {
    u = __fmul_rn(__fmul_rn(__fadd_rn(__fdiv_rn(__fsub_rn(x, h.ox), h.dx), 1.0f), 0.5f), (float)h.resx);
    v = __fmul_rn(__fmul_rn(__fadd_rn(__fdiv_rn(__fsub_rn(y, h.oy), h.dy), 1.0f), 0.5f), (float)h.resy);
}

__global__ void k_outline_mask(const float2* __restrict__ verts, const int* __restrict__ pindex, int P,
                               const int* __restrict__ edge_poly, int V, HybXf h, float margin,
                               uint32_t* __restrict__ mask, int words) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < V; k += gridDim.x * blockDim.x) {
        const int p = edge_poly[k];
        const int v0 = pindex[p], n = pindex[p + 1] - v0;
        const int kn = (k + 1 == v0 + n) ? v0 : k + 1;
        float2 A = verts[k], B = verts[kn];
        float ax, ay, bx, by;
        hyb_win(h, A.x, A.y, ax, ay);
        hyb_win(h, B.x, B.y, bx, by);
        float ylo = fminf(ay, by) - margin, yhi = fmaxf(ay, by) + margin;
        int jlo = max((int)floorf(ylo), 0), jhi = min((int)floorf(yhi), h.resy - 1);
        for (int j = jlo; j <= jhi; ++j) {
            // x extent of the segment within the slab [j - margin, j + 1 + margin]
            float sy0 = (float)j - margin, sy1 = (float)(j + 1) + margin;
            float xa, xb;
            if (ay == by) { xa = fminf(ax, bx); xb = fmaxf(ax, bx); }
            else {
                float ta = (sy0 - ay) / (by - ay), tb = (sy1 - ay) / (by - ay);
                ta = fminf(fmaxf(ta, 0.0f), 1.0f); tb = fminf(fmaxf(tb, 0.0f), 1.0f);
                float x0 = ax + (bx - ax) * ta, x1 = ax + (bx - ax) * tb;
                xa = fminf(x0, x1); xb = fmaxf(x0, x1);
            }
            int ilo = max((int)floorf(xa - margin), 0), ihi = min((int)floorf(xb + margin), h.resx - 1);
            for (int i = ilo; i <= ihi; ++i)
                atomicOr(mask + (size_t)j * words + (i >> 5), 1u << (i & 31));
        }
    }
}

// Dilation by `radius` pixels (isBorder's 3x3 neighbourhood for radius 1,
// hybrid.glsl:174-185).
__global__ void k_dilate_mask(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                              int resx, int resy, int words, int radius) {
    size_t total = (size_t)resy * words;
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < total; g += (size_t)gridDim.x * blockDim.x) {
        int j = (int)(g / words), w = (int)(g % words);
        uint32_t acc = 0;
        for (int dj = -radius; dj <= radius; ++dj) {
            int jj = j + dj;
            if (jj < 0 || jj >= resy) continue;
            const uint32_t* row = in + (size_t)jj * words;
            uint32_t c = row[w];
            uint32_t l = (w > 0) ? row[w - 1] : 0u;
            uint32_t r = (w + 1 < words) ? row[w + 1] : 0u;
            uint32_t hacc = c;
            for (int s = 1; s <= radius; ++s) {
                // bit i of out gets bits i-s and i+s of the input row
                hacc |= (c << s) | (l >> (32 - s));
                hacc |= (c >> s) | (r << (32 - s));
            }
            acc |= hacc;
        }
        out[g] = acc;
    }
}

// ---------------------------------------------------------------------------
// launchers
void launch_transform_vertices(const float2* verts, int V, const float4* colxf, const float4* rowxf,
                               int splitx, int T, int2* wv, float2* wf, int sms, cudaStream_t st) {
    size_t total = (size_t)T * V;
    int blocks = (int)std::min<size_t>((total + 255) / 256, (size_t)sms * 8);
    if (blocks < 1) blocks = 1;
    k_transform_vertices<<<blocks, 256, 0, st>>>(verts, V, colxf, rowxf, splitx, T, wv, wf);
    ++g_kernel_launches;
}

void launch_transform_vertices_xf(const float2* verts, int V, const XfArgs& col, const XfArgs& row, int splitx, int T, int2* wv,
                                  float2* wf, float4* dcol, float4* drow, int sms, cudaStream_t st) {
    const size_t total = (size_t)T * V;
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>((total + 255) / 256, (size_t)sms * 8));
    k_transform_vertices_xf<<<blocks, 256, 0, st>>>(verts, V, col, row, splitx, T, wv, wf, dcol, drow);
    ++g_kernel_launches;
}

void launch_poly_info(int mode, const PolyPassArgs& a, int sms, cudaStream_t st) {
    int items = a.T * a.P;
    int blocks = std::min((items * 32 + 255) / 256, sms * 8);
    if (blocks < 1) blocks = 1;
    ++g_kernel_launches;
    if (mode == MODE_BOUNDS) k_poly_info<MODE_BOUNDS><<<blocks, 256, 0, st>>>(a);
    else if (mode >= MODE_TIER_CLASSIFY) k_poly_info<MODE_TIER_CLASSIFY><<<blocks, 256, 0, st>>>(a);
    else k_poly_info<MODE_REDUCE><<<blocks, 256, 0, st>>>(a);
}

void launch_poly_label(const PolyPassArgs& a, int sms, cudaStream_t st) {
    ++g_kernel_launches;
    allow_smem(reinterpret_cast<const void*>(k_poly_label), kPolySmem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_poly_label, kPolyWarps * 32, kPolySmem);
    k_poly_label<<<sms * std::max(per_sm, 1), kPolyWarps * 32, kPolySmem, st>>>(a);
}

void launch_grid_count(const GridArgs& g, int sms, cudaStream_t st) {
    int blocks = std::min((g.P * 32 + 255) / 256, sms * 8);
    if (blocks < 1) blocks = 1;
    k_grid_count<<<blocks, 256, 0, st>>>(g);
    ++g_kernel_launches;
}
void launch_grid_fill(const GridArgs& g, int sms, cudaStream_t st) {
    int blocks = std::min((g.P * 32 + 255) / 256, sms * 8);
    if (blocks < 1) blocks = 1;
    k_grid_fill<<<blocks, 256, 0, st>>>(g);
    ++g_kernel_launches;
}
void launch_grid_sort(const int* cell_start, int* entries, int ncells, int sms, cudaStream_t st) {
    int blocks = std::min((ncells + 255) / 256, sms * 8);
    if (blocks < 1) blocks = 1;
    k_grid_sort<<<blocks, 256, 0, st>>>(cell_start, entries, ncells);
    ++g_kernel_launches;
}

// Scratch ints for launch_exclusive_scan: one level of tile sums per 4096x.
int scan_tmp_ints(int n) {
    int total = 0;
    int m = n;
    do {
        int ntiles = (m + kScanTile - 1) / kScanTile;
        if (ntiles < 1) ntiles = 1;
        total += ntiles + 1;
        m = ntiles;
    } while (m > kScanTile);
    return total + 1;
}

bool launch_exclusive_scan(const int* in, int* out, int n, int* tmp, cudaStream_t st) {
    // three launches cost about 7 us, one block about 1.2 us per tile of 4096
    if (n <= 4 * kScanTile) {
        k_scan_small<<<1, kScanThreads, 0, st>>>(in, out, n);
        ++g_kernel_launches;
        return true;
    }
    int ntiles = (n + kScanTile - 1) / kScanTile;
    if (ntiles < 1) ntiles = 1;
    k_scan_tiles<<<ntiles, kScanThreads, 0, st>>>(in, out, n, tmp);
    if (ntiles <= kScanTile) {
        k_scan_sums<<<1, kScanThreads, 0, st>>>(tmp, ntiles, out + n);
        g_kernel_launches += 2;
    } else {
        // scan the tile sums recursively (in place through a second buffer level)
        int* sums = tmp;
        int* next = tmp + ntiles + 1;
        if (!launch_exclusive_scan(sums, sums, ntiles, next, st)) return false;
        // out[n] = total of all tiles = scanned sums[ntiles]
        cudaMemcpyAsync(out + n, sums + ntiles, sizeof(int), cudaMemcpyDeviceToDevice, st);
        g_kernel_launches += 1;
    }
    k_scan_add<<<(n + 255) / 256, 256, 0, st>>>(out, n, tmp);
    g_kernel_launches += 1;
    return true;
}

void launch_cls_classify(const ClsArgs& c, int sms, cudaStream_t st) {
    // level 2 reads its pair count on the device; c.npairs is then an upper bound
    // A pair per lane takes about 0.38 us per edge and round of 32 pairs per warp,
    // a pair per warp 2 us and 0.007 per edge (120,000 pairs of 100 edges: 38 us
    // against 89; 20,000 pairs of jagged rings of 260: 400 against 180).
    const double slots = sms * 24.0, edges = c.edges_per_pair;
    const bool lanes = c.level != 2 && c.npairs / slots * (2.0 + 0.007 * edges) >
                                           std::max(1.0, c.npairs / (32.0 * slots)) * 0.38 * edges;
    const long long want = lanes ? ((long long)c.npairs + 127) / 128 : ((long long)c.npairs * 32 + 255) / 256;
    const int blocks = (int)std::max(1LL, std::min(want, (long long)sms * 32));
    ++g_kernel_launches;
    if (lanes) k_cls_pairs<<<blocks, 128, 0, st>>>(c);
    else k_cls_classify<<<blocks, 256, 0, st>>>(c);
}
void launch_cls_emit(const ClsArgs& c, int sms, cudaStream_t st) {
    int blocks = std::min((c.npairs + 255) / 256, sms * 16);
    if (blocks < 1) blocks = 1;
    ++g_kernel_launches;
    k_cls_emit<<<blocks, 256, 0, st>>>(c);
}
void launch_cls_fill_edges(const ClsArgs& c, int sms, cudaStream_t st) {
    int blocks = (int)std::min<long long>(((long long)c.npairs * 32 + 255) / 256, (long long)sms * 32);
    if (blocks < 1) blocks = 1;
    ++g_kernel_launches;
    k_cls_fill_edges<<<blocks, 256, 0, st>>>(c);
}
void launch_label_finish(uint16_t* label, const uint32_t* mask, int resx, int resy, int ntiles, int words,
                         unsigned long long* nonempty, int sms, cudaStream_t st) {
    size_t total = (size_t)resy * ntiles * 32;
    int blocks = (int)std::min<size_t>((total + 255) / 256, (size_t)sms * 16);
    if (blocks < 1) blocks = 1;
    ++g_kernel_launches;
    k_label_finish<<<blocks, 256, 0, st>>>(label, mask, resx, resy, ntiles, words, nonempty);
}
void launch_cls_codes(const int* cell_start, const int4* entries, uint32_t* code, int ncells, int sms,
                      cudaStream_t st) {
    int blocks = std::min((ncells + 255) / 256, sms * 16);
    if (blocks < 1) blocks = 1;
    ++g_kernel_launches;
    k_cls_codes<<<blocks, 256, 0, st>>>(cell_start, entries, code, ncells);
}

void launch_outline_mask(const float2* verts, const int* pindex, int P, const int* edge_poly, int V,
                         const HybXf& h, float margin, uint32_t* mask, int words, int sms, cudaStream_t st) {
    int blocks = std::min((V + 255) / 256, sms * 8);
    if (blocks < 1) blocks = 1;
    k_outline_mask<<<blocks, 256, 0, st>>>(verts, pindex, P, edge_poly, V, h, margin, mask, words);
    ++g_kernel_launches;
}
void launch_dilate_mask(const uint32_t* in, uint32_t* out, int resx, int resy, int words, int radius,
                        int sms, cudaStream_t st) {
    size_t total = (size_t)resy * words;
    int blocks = (int)std::min<size_t>((total + 255) / 256, (size_t)sms * 16);
    if (blocks < 1) blocks = 1;
    k_dilate_mask<<<blocks, 256, 0, st>>>(in, out, resx, resy, words, radius);
    ++g_kernel_launches;
}

}  // namespace rj
