// rj_label_core.cuh -- lean point pass of the raster join in its label form
// (polygons that do not overlap on the canvas; one canvas tile or several):
// interval-form filters on up to four columns, count or sum, into shared-
// memory histograms (points.vert:138-159 feeding polygon.frag:12-27).
//
// What bounds a label pass on GB300 is instruction issue and, when every
// point reads a block code, the L2 request rate.  Most points lie far from
// every outline, so their polygon does not depend on the exact pixel:
//   * cells: a coarse grid over the canvas, its codes in shared memory.  A
//     cell's code is the one polygon (or "none") that every pixel holds which
//     a point of the cell can fall in, the fp32 error of the pixel arithmetic
//     included, or "mixed".  The cell of a coordinate costs one FMA:
//     fma(v, a, 1.5 * 2^23 + o) rounds v * a + o to the nearest integer
//     exactly once and leaves it in the low mantissa bits, so the cells'
//     world-space edges are known exactly when the codes are built.
//     NaN, infinities and far coordinates give an index past the grid.
//   * points of mixed cells are packed into a per-warp queue in shared
//     memory and resolved 32 at a time with the exact pixel arithmetic
//     (rj_lean.cuh), the block code and the mixed block's pixel label.  The
//     two lookups are dependent L2 accesses: a batch only issues its code
//     load, the next batch's turn uses it and issues the label load, and the
//     one after that counts, so that no warp waits for them.
//   * with filters, the points that pass them are queued instead (any cell),
//     so that the lookup and histogram work runs on full warps.
// Tile seams: a cell within a pixel of a tile's edge is mixed, and the
// resolution tries every tile whose window may hold the point (within
// TileAxis::edge pixels of the edge; a point on a seam counts in each, as every tile is rendered with all points,
// RasterJoin.cpp:224-231).
//
// Measured (1B points, 260 Voronoi cells, 40000 x 40000 pixels at 1 m in 5 x 5
// tiles, count): point pass 2.10 ms, 3.8 TB/s of locations; the pass it
// replaced, one random L2 read of a block code per point and the exact pixel
// for every point, took 6.03 ms.  With a filter on four columns and avg (100M
// points, 24 B each): 0.47 ms, 5.1 TB/s.  What bounds the plain count now is
// shared-memory bandwidth (l1tex at 88 %: the code lookup and the histogram
// add of 32 random points take about three wavefronts each, the queue the
// rest), at 1.8 warp instructions per point; exact pixels for every point
// took 3.1.  About 64k cells (128 KB of codes, one block of 1024 threads per
// SM) beat 16k with more blocks: fewer points are queued (23 % against 35 %).
// Far from the origin fp32 places points off by whole pixels.  Beyond half a
// pixel (1 m tiles of 8,000 pixels: from some 700,000 pixels from the origin) no
// cell is uniform and every point takes the queue: 400M points at 1 m, 2.29 ms
// with y = 4.1e6 (UTM) or x = -8.2e6 (Web Mercator), 1.27 at the origin, 3.02
// with the pass before at any of them.  At 10 m, or with filters, the times are
// the same.
#pragma once
#include "rj_lean.cuh"

namespace rj {

constexpr int kLeanMaxSplit = 64;   // canvas tiles per axis held in shared memory

// ---- tiles ------------------------------------------------------------------
// Tiles [lo, hi] of one axis whose window may hold coordinate v (lo > hi: none).
__device__ __forceinline__ void tl_range(float v, int split, float lb, float inv_td, int& lo, int& hi) {
    lo = 0;
    hi = 0;
    if (split == 1) return;
    const float g = (v - lb) * inv_td;
    if (!(g > -2.0f && g < (float)split + 1.0f)) {   // NaN, infinities, far outside
        hi = -1;
        return;
    }
    const int c = (int)floorf(g);
    lo = max(c - 1, 0);
    hi = min(c + 1, split - 1);
}

// The tiles of an axis have one extent, so they share the scale s and the half
// resolution (the launching code checks it); only the offset t[c] differs.
// One axis: v's pixel in tile c.
__device__ __forceinline__ int tl_pixel(float v, const TileAxis& x, const float* t, int c) {
    return snapped_pixel(v, x.s, t[c], x.H);
}

// The common case of one axis: the guessed tile c holds v far enough inside its
// window, in pixel q, that no other tile does.
__device__ __forceinline__ bool tl_inner(float v, const TileAxis& x, const float* t, int& c, int& q) {
    c = __float2int_rd((v - x.lb) * x.inv_td);
    const bool guess = (unsigned)c < (unsigned)x.split;
    c = guess ? c : 0;
    q = tl_pixel(v, x, t, c);
    return guess && q >= x.edge && q < x.res - x.edge;
}

// Every (tile, pixel) of a point: f(tile column, tile row, px, py).
template <class F>
__device__ __forceinline__ void tl_hits(const TileAxis& ax, const TileAxis& ay, const float* tx, const float* ty, float x,
                                        float y, F&& f) {
    int x0, x1, y0, y1;
    tl_range(x, ax.split, ax.lb, ax.inv_td, x0, x1);
    tl_range(y, ay.split, ay.lb, ay.inv_td, y0, y1);
    #pragma unroll 1
    for (int cy = y0; cy <= y1; ++cy) {
        const int py = tl_pixel(y, ay, ty, cy);
        if ((unsigned)py >= (unsigned)ay.res) continue;
        #pragma unroll 1
        for (int cx = x0; cx <= x1; ++cx) {
            const int px = tl_pixel(x, ax, tx, cx);
            if ((unsigned)px < (unsigned)ax.res) f(cx, cy, px, py);
        }
    }
}

// The tile offsets into shared memory.
template <int BLOCK>
__device__ __forceinline__ void tl_stage_tiles(const TileAxis& ax, const TileAxis& ay, float* tx, float* ty) {
    for (int i = threadIdx.x; i < ax.split; i += BLOCK) tx[i] = __ldg(ax.xf + i).y;
    for (int i = threadIdx.x; i < ay.split; i += BLOCK) ty[i] = __ldg(ay.xf + i).y;
}

// Whether a zone of the warp's 64 * NV rows meets the query's reach (no zone
// map: yes).
template <int NV, class A>
__device__ __forceinline__ bool tl_zone(const A& a, uint64_t first_pair) {
    if (!a.zones) return true;
    const uint64_t r0 = a.zrow0 + 2 * first_pair;
    const uint64_t r1 = a.zrow0 + min(2 * (first_pair + 32 * NV), a.n) - 1;
    const int lane = threadIdx.x & 31;
    bool meets = false;
    if (r0 <= r1 && (uint64_t)lane <= (r1 >> kZoneShift) - (r0 >> kZoneShift)) {
        const float4 b = __ldg(a.zones + (r0 >> kZoneShift) + lane);
        meets = !(b.z < a.qbox.x || b.x > a.qbox.z || b.w < a.qbox.y || b.y > a.qbox.w);
    }
    return __any_sync(0xffffffffu, meets);
}

// ---- filters and sums ---------------------------------------------------------
// The predicates of a point: the first NI columns hold uint / int values, the
// next NF floats (LeanCols: key - lo <= span, key = v or v ^ (sign(v) & 2^31-1)).
template <int NI, int NF>
__device__ __forceinline__ bool cols_pass(const LeanCols& lc, const uint32_t* v) {
    bool ok = true;
    #pragma unroll
    for (int c = 0; c < NI + NF; ++c) {
        const uint32_t key = c < NI ? v[c] : v[c] ^ ((uint32_t)((int32_t)v[c] >> 31) & 0x7FFFFFFFu);
        ok &= (key - lc.lo[c]) <= lc.span[c];
    }
    return ok;
}

// One point of polygon l into a histogram copy: count | sum low | sum high.
template <bool AGG>
__device__ __forceinline__ void label_add(uint32_t* hist, uint32_t P, const LeanCols& lc, uint32_t l, float v) {
    atomicAdd(hist + l, 1u);
    if (AGG) {
        if (isfinite(v)) {
            const unsigned long long q = (unsigned long long)fixed_value(v, lc.scale);
            const uint32_t qlo = (uint32_t)q;
            const uint32_t old = atomicAdd(hist + P + l, qlo);
            atomicAdd(hist + 2 * P + l, (uint32_t)(q >> 32) + ((old + qlo < old) ? 1u : 0u));
        } else {
            atomicAdd(lc.nonfinite + l, (double)v);
        }
    }
}

// The block's histogram copies into the outputs.
template <int BLOCK, bool AGG>
__device__ __forceinline__ void label_flush(const LabelPointArgs& a, const LeanCols& lc, const uint32_t* s_hist) {
    constexpr int HW = AGG ? 3 : 1;
    for (int b = threadIdx.x; b < a.P; b += BLOCK) {
        uint32_t cnt = 0;
        unsigned long long sum = 0;
        #pragma unroll 1
        for (int w = 0; w < lc.copies; ++w) {
            const uint32_t* h = s_hist + w * HW * a.P;
            cnt += h[b];
            if (AGG) sum += ((unsigned long long)h[2 * a.P + b] << 32) + h[a.P + b];
        }
        if (cnt) {
            atomicAdd(a.out_count + b, (unsigned long long)cnt);
            if (AGG) atomicAdd(lc.out_sum + b, sum);
        }
    }
}

// ---- the pass -------------------------------------------------------------------
template <int BLOCK, int NV, int MINB, int NI, int NF, bool AGG>
__global__ void __launch_bounds__(BLOCK, MINB) k_label_points(LabelPointArgs a, LeanCols lc) {
    extern __shared__ uint32_t s_words[];
    constexpr int HW = AGG ? 3 : 1;
    constexpr int NCOL = NI + NF;
    constexpr int NA = NCOL > 0 ? NCOL : 1;
    constexpr int G = NV < 2 ? NV : 2;       // pairs queued at a time
    constexpr int QC = 32 + 64 * G;          // queued points of a warp: fewer than 32 left over plus one group's
    float* tx = reinterpret_cast<float*>(s_words);
    float* ty = tx + kLeanMaxSplit;
    float2* s_q = reinterpret_cast<float2*>(ty + kLeanMaxSplit);      // queued locations, QC per warp
    uint32_t* s_qv = reinterpret_cast<uint32_t*>(s_q + (BLOCK / 32) * QC);   // AGG: their values (raw)
    uint32_t* s_code = s_qv + (AGG ? (BLOCK / 32) * QC : 0);
    uint32_t* s_hist = s_code + a.cell_words;                         // lc.copies x HW x P
    tl_stage_tiles<BLOCK>(a.ax, a.ay, tx, ty);
    {
        const uint32_t* g = reinterpret_cast<const uint32_t*>(a.cells);
        for (int i = threadIdx.x; i < a.cell_words; i += BLOCK) s_code[i] = __ldg(g + i);
        for (int i = threadIdx.x; i < lc.copies * HW * a.P; i += BLOCK) s_hist[i] = 0u;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint16_t* sc = reinterpret_cast<const uint16_t*>(s_code);
    const uint32_t P = (uint32_t)a.P;
    uint32_t* hist = s_hist + (warp & (lc.copies - 1)) * HW * a.P;
    float2* q = s_q + warp * QC;
    uint32_t* qv = s_qv + warp * QC;
    int qn = 0;                                                       // queued points (warp-uniform)

    auto cell_code = [&](float x, float y) -> uint32_t {
        const uint32_t ix = __float_as_uint(fmaf(x, a.cax, a.ccx)) - kCellMagic;
        const uint32_t iy = __float_as_uint(fmaf(y, a.cay, a.ccy)) - kCellMagic;
        // the last column and row hold "none": indices past the grid land there
        return sc[min(iy, (uint32_t)a.cny) * (uint32_t)(a.cnx + 1) + min(ix, (uint32_t)a.cnx)];
    };
    // a point of a mixed cell near a tile's edge (or off the canvas): every hit
    auto resolve_edge = [&](float x, float y, float v) {
        tl_hits(a.ax, a.ay, tx, ty, x, y, [&](int cx, int cy, int px, int py) {
            uint32_t l = __ldg(a.tr.code + ((cy * a.ax.split + cx) * a.tr.bh + (py >> 4)) * a.tr.bw + (px >> 4));
            if (l >= kTierMixed && l < kTierMulti)
                l = __ldg(a.tr.plabel + (size_t)(l & ~kTierMixed) * 256 + ((py & 15) << 4 | (px & 15)));
            if (l < P) label_add<AGG>(hist, P, lc, l, v);
        });
    };
    // batches in flight: the last one's block code, the one before's label
    uint32_t code1 = kTierEmpty, ofs1 = 0u, lab2 = kTierEmpty;
    float val1 = 0.f, val2 = 0.f;
    auto advance = [&]() {
        if (lab2 < P) label_add<AGG>(hist, P, lc, lab2, val2);
        lab2 = code1;
        val2 = val1;
        if (code1 >= kTierMixed && code1 < kTierMulti)
            lab2 = __ldg(a.tr.plabel + (size_t)(code1 & ~kTierMixed) * 256 + ofs1);
        code1 = kTierEmpty;
    };
    // the last 32 (or fewer) queued points
    auto drain = [&]() {
        advance();
        const int first = max(qn - 32, 0);
        const int i = first + lane;
        if (i < qn) {
            const float2 p = q[i];
            const float v = AGG ? agg_value(lc.aggr_typ, qv[i]) : 0.f;
            uint32_t l = kCodeMixed;
            if (NCOL > 0) {
                l = cell_code(p.x, p.y);
                if (l < P) label_add<AGG>(hist, P, lc, l, v);
            }
            if (l == kCodeMixed) {
                int cx, cy, px, py;
                if (tl_inner(p.x, a.ax, tx, cx, px) & tl_inner(p.y, a.ay, ty, cy, py)) {
                    code1 = __ldg(a.tr.code + ((cy * a.ax.split + cx) * a.tr.bh + (py >> 4)) * a.tr.bw + (px >> 4));
                    ofs1 = (py & 15) << 4 | (px & 15);
                    val1 = v;
                } else {
                    resolve_edge(p.x, p.y, v);
                }
            }
        }
        qn = first;
        __syncwarp();
    };

    const uint64_t npairs = a.n >> 1;
    constexpr uint64_t kPerIter = (uint64_t)BLOCK * NV;
    const uint64_t warp_ofs = (uint64_t)warp * 32 * NV;
    auto iterate = [&](uint64_t base, bool full) {
        float4 p[NV];
        uint2 cv[NA][NV];
        uint2 av[NV];
        #pragma unroll
        for (int k = 0; k < NV; ++k) {
            const uint64_t i = base + warp_ofs + lane + (uint64_t)k * 32;
            const bool live = full || i < npairs;
            p[k] = live ? __ldcs(a.xy + i) : make_float4(NAN, NAN, NAN, NAN);
            #pragma unroll
            for (int c = 0; c < NCOL; ++c) cv[c][k] = live ? __ldcs(lc.col[c] + i) : make_uint2(0u, 0u);
            if (AGG) av[k] = (live && lc.aggr_ci < 0) ? __ldcs(lc.aggr_col + i) : make_uint2(0u, 0u);
        }
        auto value = [&](int j) -> uint32_t {
            uint32_t raw = (j & 1) ? av[j >> 1].y : av[j >> 1].x;
            #pragma unroll
            for (int c = 0; c < NCOL; ++c)
                if (c == lc.aggr_ci) raw = (j & 1) ? cv[c][j >> 1].y : cv[c][j >> 1].x;
            return raw;
        };
        #pragma unroll
        for (int g = 0; g < NV; g += G) {
            uint32_t push = 0u;   // points to queue: survivors of the filters, or points of mixed cells
            #pragma unroll
            for (int j = 2 * g; j < 2 * (g + G); ++j) {
                if (NCOL > 0) {
                    uint32_t v[NA];
                    #pragma unroll
                    for (int c = 0; c < NCOL; ++c) v[c] = (j & 1) ? cv[c][j >> 1].y : cv[c][j >> 1].x;
                    bool ok = cols_pass<NI, NF>(lc, v);
                    if (!full) ok = ok && base + warp_ofs + lane + (uint64_t)(j >> 1) * 32 < npairs;
                    push |= ok ? 1u << j : 0u;
                } else {
                    const uint32_t l =
                        cell_code((j & 1) ? p[j >> 1].z : p[j >> 1].x, (j & 1) ? p[j >> 1].w : p[j >> 1].y);
                    if (l < P) label_add<AGG>(hist, P, lc, l, AGG ? agg_value(lc.aggr_typ, value(j)) : 0.f);
                    push |= l == kCodeMixed ? 1u << j : 0u;
                }
            }
            // queue positions: one prefix sum over the lanes for the group
            int incl = __popc(push);
            const int own = incl;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            int at = qn + incl - own;
            #pragma unroll
            for (int j = 2 * g; j < 2 * (g + G); ++j)
                if ((push >> j) & 1u) {
                    q[at] = (j & 1) ? make_float2(p[j >> 1].z, p[j >> 1].w) : make_float2(p[j >> 1].x, p[j >> 1].y);
                    if (AGG) qv[at] = value(j);
                    ++at;
                }
            qn += __shfl_sync(0xffffffffu, incl, 31);
            __syncwarp();
            while (qn >= 32) drain();
        }
    };
    for (uint64_t base = (uint64_t)blockIdx.x * kPerIter; base < npairs; base += (uint64_t)gridDim.x * kPerIter) {
        if (!tl_zone<NV>(a, base + warp_ofs)) continue;
        if (base + kPerIter <= npairs) iterate(base, true);
        else iterate(base, false);
    }
    if (qn > 0) drain();
    advance();
    advance();
    // the last point of an odd-sized table
    if ((a.n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const uint64_t i = a.n - 1;
        const float2 p = __ldg(reinterpret_cast<const float2*>(a.xy) + i);
        uint32_t v[NA];
        #pragma unroll
        for (int c = 0; c < NCOL; ++c) v[c] = __ldg(reinterpret_cast<const uint32_t*>(lc.col[c]) + i);
        if (cols_pass<NI, NF>(lc, v)) {
            float fv = 0.f;
            if (AGG) {
                uint32_t raw = lc.aggr_ci < 0 ? __ldg(reinterpret_cast<const uint32_t*>(lc.aggr_col) + i) : 0u;
                #pragma unroll
                for (int c = 0; c < NCOL; ++c)
                    if (c == lc.aggr_ci) raw = v[c];
                fv = agg_value(lc.aggr_typ, raw);
            }
            resolve_edge(p.x, p.y, fv);
        }
    }
    __syncthreads();
    label_flush<BLOCK, AGG>(a, lc, s_hist);
}

// Shapes: threads, point pairs in flight per thread, blocks per SM the
// registers allow.
struct LabelShape {
    int block, nv, minb;
};
constexpr LabelShape kLabelShapes[] = {{1024, 4, 1}, {1024, 2, 1}, {512, 2, 3}};
constexpr int kNumLabelShapes = (int)(sizeof(kLabelShapes) / sizeof(kLabelShapes[0]));

using LabelKernel = void (*)(LabelPointArgs, LeanCols);
// launches a label kernel on as many blocks as are resident (fewer for short
// scans); false when it cannot run, nothing launched
bool launch_label_kernel(LabelKernel k, int block, int nv, size_t smem, const LabelPointArgs& a, const LeanCols& lc,
                         int sms, cudaStream_t st);
LabelKernel label_points_count(int shape, int ni, int nf);   // rj_label_count.cu
LabelKernel label_points_sum(int shape, int ni, int nf);     // rj_label_sum.cu

template <int NI, int NF, bool AGG>
LabelKernel label_kernel(int shape) {
    switch (shape) {
        case 0: return k_label_points<1024, 4, 1, NI, NF, AGG>;
        case 1: return k_label_points<1024, 2, 1, NI, NF, AGG>;
        case 2: return k_label_points<512, 2, 3, NI, NF, AGG>;
        default: return nullptr;
    }
}

template <bool AGG>
LabelKernel label_kernel_cols(int shape, int ni, int nf) {
    switch (ni * 5 + nf) {
        case 0: return label_kernel<0, 0, AGG>(shape);
        case 1: return label_kernel<0, 1, AGG>(shape);
        case 2: return label_kernel<0, 2, AGG>(shape);
        case 3: return label_kernel<0, 3, AGG>(shape);
        case 4: return label_kernel<0, 4, AGG>(shape);
        case 5: return label_kernel<1, 0, AGG>(shape);
        case 6: return label_kernel<1, 1, AGG>(shape);
        case 7: return label_kernel<1, 2, AGG>(shape);
        case 8: return label_kernel<1, 3, AGG>(shape);
        case 10: return label_kernel<2, 0, AGG>(shape);
        case 11: return label_kernel<2, 1, AGG>(shape);
        case 12: return label_kernel<2, 2, AGG>(shape);
        case 15: return label_kernel<3, 0, AGG>(shape);
        case 16: return label_kernel<3, 1, AGG>(shape);
        case 20: return label_kernel<4, 0, AGG>(shape);
        default: return nullptr;
    }
}

}  // namespace rj
