// rj_band_kernels.cu -- the polygon passes that read a point canvas: the sum
// over every polygon's covered pixels (polygon.frag:12-27) and the error-bound
// outline pass (line-bound.frag:243-286).
//
// A polygon's covered pixels of a row are spans between its crossings with the
// row's centre line, so with the canvas rows replaced by their prefix sums
// (k_row_prefix) a span costs two reads whatever its length: the pass follows
// the polygons' perimeters, not their areas.
//
// k_poly_bands: one warp per (tile, polygon, band of 16 rows).
//   * the band's edges are staged in shared memory;
//   * the (edge, row) crossings of the whole band are spread over the lanes
//     (one exact crossing each) and kept in lists, one per row;
//   * spans: the sorted crossings c0 <= c1 <= ... of a row bound the spans
//     [c0, c1), [c2, c3), ...; a crossing's contribution to the sum is its
//     prefix with the sign of its rank's parity, which the lane finds by
//     comparing with the row's others -- no sorting, no order between lanes;
//   * outline: the (edge, row) pairs are spread the same way; a lane takes the
//     few pixels of its pair (a wide pair is taken by the whole warp) and reads
//     their counts together; the pixels that hold points are packed into a
//     queue and clipped 32 at a time; whether a pixel centre lies inside is the
//     parity of the row's crossings right of it.
//
// Measured: 2,000 stars on 4000 x 4000 pixels, prefix sums and spans 0.22 ms
// where a pass over the areas took 0.45; the outlines of 2,000 stars at 1 m
// (40,000 x 40,000 pixels) 6.0 ms, 15.8 before.  What bounds both is latency: a
// band is a chain of staging, crossings and reads, and 24 to 32 warps per SM are
// resident.  The row prefix of 4000 x 4000 counts takes 31 us, 4.1 TB/s.
#include <climits>

#include "rj_bands.cuh"
#include "rj_launch.h"

namespace rj {

namespace {

// ---------------------------------------------------------------------------
// Rows of the canvas -> inclusive prefix sums: counts in place (or into 64
// bits, for tables of 2^32 rows and more), fixed-point sums in place (modulo
// 2^64).  One block per row, four pixels per thread and step.
constexpr int kPrefixThreads = 256;

template <class T>
__device__ __forceinline__ T block_scan(T v, T* s_warp, T& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    T base = 0;
    total = 0;
    #pragma unroll
    for (int w = 0; w < kPrefixThreads / 32; ++w) {
        const T s = s_warp[w];
        base += w < warp ? s : T(0);
        total += s;
    }
    __syncthreads();
    return base + x;   // inclusive
}

template <class IN, class OUT>
__device__ __forceinline__ void prefix_row(const IN* in, OUT* out, int n, OUT* s_warp) {
    OUT carry = 0;
    for (int x0 = 0; x0 < n; x0 += kPrefixThreads * 4) {
        const int x = x0 + (int)threadIdx.x * 4;
        OUT v[4];
        #pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = x + i < n ? (OUT)in[x + i] : OUT(0);
        #pragma unroll
        for (int i = 1; i < 4; ++i) v[i] += v[i - 1];
        OUT total;
        const OUT before = carry + block_scan<OUT>(v[3], s_warp, total) - v[3];
        #pragma unroll
        for (int i = 0; i < 4; ++i)
            if (x + i < n) out[x + i] = before + v[i];
        carry += total;
    }
}

__global__ void __launch_bounds__(kPrefixThreads) k_row_prefix(uint32_t* c, unsigned long long* wide, unsigned long long* s,
                                                               int resx, int rows) {
    __shared__ unsigned long long s_warp[kPrefixThreads / 32];
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const size_t at = (size_t)r * resx;
        if (wide) prefix_row(c + at, wide + at, resx, s_warp);
        else prefix_row(c + at, c + at, resx, reinterpret_cast<uint32_t*>(s_warp));
        if (s) prefix_row(s + at, s + at, resx, s_warp);
    }
}

// ---------------------------------------------------------------------------
// Cohen-Sutherland clip of an edge against one pixel and the area fraction on
// one side, computeFraction line-bound.frag:51-211, in fp32 window units.
__device__ __forceinline__ int cs_outcode(float x, float y, float xmin, float ymin, float xmax, float ymax) {
    int code = 0;
    if (x < xmin) code |= 1;
    else if (x > xmax) code |= 2;
    if (y < ymin) code |= 4;
    else if (y > ymax) code |= 8;
    return code;
}

__device__ __forceinline__ float tri_area(float ax, float ay, float bx, float by, float cx, float cy) {
    // abs(0.5 * length(cross(b - a, c - a))) with z = 0
    float ix = __fsub_rn(bx, ax), iy = __fsub_rn(by, ay);
    float jx = __fsub_rn(cx, ax), jy = __fsub_rn(cy, ay);
    float cz = __fsub_rn(__fmul_rn(ix, jy), __fmul_rn(iy, jx));
    return fabsf(__fmul_rn(0.5f, cz));
}

__device__ bool compute_fraction(float x0, float y0, float x1, float y1,
                                 float xmin, float ymin, float xmax, float ymax, float& frac) {
    int oc0 = cs_outcode(x0, y0, xmin, ymin, xmax, ymax);
    int oc1 = cs_outcode(x1, y1, xmin, ymin, xmax, ymax);
    bool accept = false;
    frac = 0.0f;
    for (int it = 0; it < 16; ++it) {   // the reference loops until accept/reject
        if ((oc0 | oc1) == 0) { accept = true; break; }
        if ((oc0 & oc1) != 0) break;
        float x = 0.0f, y = 0.0f;
        int out = (oc0 != 0) ? oc0 : oc1;
        if (out & 8) {
            x = __fadd_rn(x0, __fdiv_rn(__fmul_rn(__fsub_rn(x1, x0), __fsub_rn(ymax, y0)), __fsub_rn(y1, y0)));
            y = ymax;
        } else if (out & 4) {
            x = __fadd_rn(x0, __fdiv_rn(__fmul_rn(__fsub_rn(x1, x0), __fsub_rn(ymin, y0)), __fsub_rn(y1, y0)));
            y = ymin;
        } else if (out & 2) {
            y = __fadd_rn(y0, __fdiv_rn(__fmul_rn(__fsub_rn(y1, y0), __fsub_rn(xmax, x0)), __fsub_rn(x1, x0)));
            x = xmax;
        } else if (out & 1) {
            y = __fadd_rn(y0, __fdiv_rn(__fmul_rn(__fsub_rn(y1, y0), __fsub_rn(xmin, x0)), __fsub_rn(x1, x0)));
            x = xmin;
        }
        if (out == oc0) { x0 = x; y0 = y; oc0 = cs_outcode(x0, y0, xmin, ymin, xmax, ymax); }
        else            { x1 = x; y1 = y; oc1 = cs_outcode(x1, y1, xmin, ymin, xmax, ymax); }
    }
    if (!accept) return false;
    if (x0 > x1) { float t = x0; x0 = x1; x1 = t; t = y0; y0 = y1; y1 = t; }
    float v1x = 0, v1y = 0, v2x = 0, v2y = 0, v3x = 0, v3y = 0, v4x = 0, v4y = 0;
    bool tri = false, compute = true;
    if (x0 == xmin) {
        if (x1 == xmax) {                      // horizontal cut
            v1x = xmin; v1y = ymin; v2x = xmax; v2y = ymin; v3x = x1; v3y = y1; v4x = x0; v4y = y0;
        } else if (y1 == ymax) {
            v1x = xmin; v1y = ymax; v2x = x0; v2y = y0; v3x = x1; v3y = y1; tri = true;
        } else if (y1 == ymin) {
            v1x = xmin; v1y = ymin; v2x = x0; v2y = y0; v3x = x1; v3y = y1; tri = true;
        } else {
            compute = false;
        }
    } else if (x1 == xmax) {
        if (y0 == ymax) {
            v1x = xmax; v1y = ymax; v2x = x0; v2y = y0; v3x = x1; v3y = y1; tri = true;
        } else if (y0 == ymin) {
            v1x = xmax; v1y = ymin; v2x = x1; v2y = y1; v3x = x0; v3y = y0; tri = true;
        } else {
            compute = false;
        }
    } else if (y0 == ymin && y1 == ymax) {     // vertical cut
        v1x = xmin; v1y = ymin; v2x = xmin; v2y = ymax; v3x = x1; v3y = y1; v4x = x0; v4y = y0;
    } else if (y1 == ymin && y0 == ymax) {     // vertical cut
        v1x = xmin; v1y = ymin; v2x = xmin; v2y = ymax; v3x = x0; v3y = y0; v4x = x1; v4y = y1;
    } else {
        compute = false;
    }
    frac = 0.5f;
    if (compute) {
        float area = tri_area(v1x, v1y, v2x, v2y, v3x, v3y);
        if (!tri) area = __fadd_rn(area, tri_area(v1x, v1y, v3x, v3y, v4x, v4y));
        frac = __fdiv_rn(area, __fmul_rn(__fsub_rn(ymax, ymin), __fsub_rn(xmax, xmin)));
    }
    return true;
}

// ---------------------------------------------------------------------------
constexpr int kBW = 8;             // warps per block
constexpr int kBEdges = 128;       // staged edges per warp
constexpr int kBCross = 512;       // crossings held per warp (rows of the band taken in groups that fit)
// Bits of a column beside the four of a band's row.  A hybrid canvas can be far
// wider than a raster tile's 8192 pixels; from 31 * 2^22 columns on its border
// radius, at least columns * 2^-22, is refused.
constexpr int kColBits = 28;
constexpr uint32_t kColMask = (1u << kColBits) - 1u;
static_assert(kBand <= 1 << (32 - kColBits), "a band's rows fit beside the column");

struct BandWarp {
    int4 edge[kBEdges];
    int eidx[kBEdges];
    uint32_t cross[kBCross];       // crossing column, clamped to the polygon's columns, | row << kColBits
    int start[kBand + 1];          // first crossing of each row
    int cur[kBand];                // crossings of each row
};
// outline: pixels that hold points, waiting for their clip (vertex, column |
// row << 16, count); fewer than 32 left over plus four of every lane
struct OutlineQueue {
    int k[160];
    uint32_t at[160];
    uint32_t val[160];
};
static_assert(sizeof(BandWarp) % 16 == 0, "BandWarp keeps 16-byte alignment");

template <bool SPANS, bool OUTLINE, class C>
__global__ void __launch_bounds__(kBW * 32, OUTLINE ? 3 : 4) k_poly_bands(PolyPassArgs a, const C* __restrict__ prefix) {
    __shared__ BandWarp s_band[kBW];
    __shared__ OutlineQueue s_queue[OUTLINE ? kBW : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    const int TP = a.T * a.P;
    BandWarp& S = s_band[warp];
    BandItems work(a.band_start, TP, a.work_ctr, kBW, warp, lane);

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
        const float2* pf = OUTLINE ? a.wf + (size_t)t * a.V + v0 : nullptr;
        const size_t row0 = ((size_t)t * a.resy + jb) * a.resx;   // first pixel of the band's first row

        // edges within a pixel of the band's rows
        const int64_t band_lo = (int64_t)jb * kSub - kSub;
        const int64_t band_hi = (int64_t)(je + 1) * kSub + kSub;
        const int nb = stage_edges(pv, n, band_lo, band_hi, lane, [&](int pos, int k, const int4& e) {
            if (pos < kBEdges) {
                S.edge[pos] = e;
                if (OUTLINE) S.eidx[pos] = k;
            }
        });
        const bool overflow = nb > kBEdges;
        const int ne = overflow ? n : nb;
        auto edge_at = [&](int e) -> int4 {
            if (!overflow) return S.edge[e];
            const int2 A = pv[e];
            const int2 B = pv[(e + 1 == n) ? 0 : e + 1];
            return make_int4(A.x, A.y, B.x, B.y);
        };
        // crossings per row (rows whose centre the polygon can cross)
        const int cl = max(j_lo, jb) - jb, ch = min(j_hi, je) - jb;
        if (lane <= kBand) S.start[lane] = 0;
        __syncwarp();
        for (int e = lane; e < ne; e += 32) {
            const int4 q = edge_at(e);
            int r0, r1;
            edge_rows(q.y, q.w, jb, r0, r1);
            r0 = max(r0, cl);
            r1 = min(r1, ch);
            if (r0 <= r1) {
                atomicAdd(&S.start[r0], 1);
                atomicAdd(&S.start[r1 + 1], -1);
            }
        }
        __syncwarp();
        unsigned pairs = 0;   // of crossings in one row
        int most = 0;         // crossings of a row
        {
            // differences -> counts -> first crossing of each row
            int c = lane < kBand ? S.start[lane] : 0;
            #pragma unroll
            for (int o = 1; o < kBand; o <<= 1) {
                const int v = __shfl_up_sync(FULL, c, o);
                if (lane >= o) c += v;
            }
            int x = lane < kBand ? c : 0;
            most = __reduce_max_sync(FULL, x);
            pairs = __reduce_add_sync(FULL, (unsigned)min(x, 4096) * (unsigned)min(x, 4096));
            #pragma unroll
            for (int o = 1; o < kBand; o <<= 1) {
                const int v = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += v;
            }
            __syncwarp();
            if (lane < kBand) S.start[lane + 1] = x;
            if (lane == 0) S.start[0] = 0;
        }
        __syncwarp();

        unsigned long long acc_c = 0, acc_s = 0;
        long long b_fn = 0, b_fp = 0, b_fn1 = 0, b_fp1 = 0;
        const int nrows = je - jb + 1;
        // Rows with few crossings rank each against the others.  Where that is
        // dearer, a row is a bitmap instead, one bit per column, a crossing
        // flipping its bit: the parity of the bits left of it is its rank's, and
        // as a ring crosses a row an even number of times, one running parity
        // serves all rows of a group.  About 6 instructions per pair against 25
        // per word and 60 per edge and group of rows, each for 32 at a time.  On
        // ten rings of up to 2,000 vertices, 1192 x 1137 pixels, 83 us; 784 with
        // ranks and a test of every pixel in rows of more than 512 crossings.
        // (Not in the outline pass: the code for both made it spill, 2,000 stars
        // and 200M points at 1 m took 19.2 ms instead of 15.7.)
        const int width = i_lo <= i_hi ? (i_hi - i_lo + 2 + 31) >> 5 : 0;   // words of a row
        const int fit = width > 0 ? kBCross / width : 0;                    // rows of a group
        const bool bits = !OUTLINE && fit > 0 && (most > kBCross || pairs > 4u * (unsigned)(nrows * width) +
                                                                    10u * (unsigned)((nrows + fit - 1) / fit * ne));
        // inside test over every edge (a row with more crossings than are held)
        auto inside_slow = [&](int i, int r) {
            const int32_t cy = (jb + r) * kSub + kSub / 2;
            bool in = false;
            for (int k = 0; k < n; ++k) {
                const int2 A = pv[k];
                const int2 B = pv[(k + 1 == n) ? 0 : k + 1];
                if (cross_row(A.y, B.y, cy)) in ^= (i < cross_L(A.x, A.y, B.x, B.y, cy));
            }
            return in;
        };
        auto prefix_at = [&](int r, int x) -> C {   // sum of the row's pixels [0, x)
            return x > 0 ? __ldg(prefix + row0 + (size_t)r * a.resx + x - 1) : C(0);
        };

        for (int ra = 0; ra < nrows;) {
            int rb = ra + 1;
            if (bits) rb = min(ra + fit, nrows);
            else
                while (rb < nrows && S.start[rb + 1] - S.start[ra] <= kBCross) ++rb;
            const int base = S.start[ra], m = S.start[rb] - base;
            const bool slow = !bits && m > kBCross;   // then one row
            if (lane < kBand) S.cur[lane] = 0;
            if (bits)
                for (int w = lane; w < (rb - ra) * width; w += 32) S.cross[w] = 0u;
            __syncwarp();
            if (m > 0 && bits) {
                for_edge_rows(ne, jb, lane, edge_at, [&](const int4& q, int r) {
                    const int32_t cy = (jb + r) * kSub + kSub / 2;
                    if (r < max(ra, cl) || r >= rb || r > ch || !cross_row(q.y, q.w, cy)) return;
                    const int b = min(max(cross_L(q.x, q.y, q.z, q.w, cy), i_lo), i_hi + 1) - i_lo;
                    atomicXor(&S.cross[(r - ra) * width + (b >> 5)], 1u << (b & 31));
                });
                __syncwarp();
                unsigned carry = 0u;
                for (int w0 = 0; w0 < (rb - ra) * width; w0 += 32) {
                    const int w = w0 + lane;
                    unsigned t = w < (rb - ra) * width ? S.cross[w] : 0u;
                    const unsigned odd = __ballot_sync(FULL, __popc(t) & 1);
                    unsigned before = (__popc(odd & ((1u << lane) - 1u)) ^ carry) & 1u;
                    carry ^= __popc(odd) & 1u;
                    const int r = ra + w / width, x0 = i_lo + (w % width) * 32;
                    while (__any_sync(FULL, t != 0u)) {
                        C c[4];
                        unsigned long long cs[4];
                        bool plus[4];
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int L = t ? x0 + __ffs(t) - 1 : 0;   // (nothing is left of column 0)
                            plus[u] = before != 0u;
                            before ^= t ? 1u : 0u;
                            t &= t - 1;
                            c[u] = prefix_at(r, L);
                            cs[u] = a.canvas_s && L > 0
                                        ? (unsigned long long)__ldg(a.canvas_s + row0 + (size_t)r * a.resx + L - 1) : 0ull;
                        }
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            acc_c += plus[u] ? (unsigned long long)c[u] : 0ull - c[u];
                            acc_s += plus[u] ? cs[u] : 0ull - cs[u];
                        }
                    }
                }
            } else if (m > 0 && !slow) {
                for_edge_rows(ne, jb, lane, edge_at, [&](const int4& q, int r) {
                    const int32_t cy = (jb + r) * kSub + kSub / 2;
                    if (r < max(ra, cl) || r >= rb || r > ch || !cross_row(q.y, q.w, cy)) return;
                    const int L = max(min(max(cross_L(q.x, q.y, q.z, q.w, cy), i_lo), i_hi + 1), 0);
                    S.cross[S.start[r] - base + atomicAdd(&S.cur[r], 1)] = (uint32_t)L | ((uint32_t)r << kColBits);
                });
            }
            __syncwarp();
            if (SPANS && !bits && m > 0 && i_lo <= i_hi) {
                if (!slow) {
                    for (int x = lane; x < m; x += 32) {
                        const uint32_t mine = S.cross[x];
                        const int r = (int)(mine >> kColBits), L = (int)(mine & kColMask);
                        const int f = S.start[r] - base, e = f + S.cur[r];
                        bool odd = false;
                        for (int k = f; k < e; ++k) {
                            const uint32_t o = S.cross[k];
                            odd ^= o < mine || (o == mine && k < x);
                        }
                        const unsigned long long c = prefix_at(r, L);
                        acc_c += odd ? c : 0ull - c;
                        if (a.canvas_s && L > 0) {
                            const unsigned long long s =
                                (unsigned long long)__ldg(a.canvas_s + row0 + (size_t)r * a.resx + L - 1);
                            acc_s += odd ? s : 0ull - s;
                        }
                    }
                } else {
                    for (int i = i_lo + lane; i <= i_hi; i += 32)
                        if (inside_slow(i, ra)) {
                            acc_c += (unsigned long long)(C)(prefix_at(ra, i + 1) - prefix_at(ra, i));
                            if (a.canvas_s) {
                                const long long* s = a.canvas_s + row0 + (size_t)ra * a.resx + i;
                                acc_s += (unsigned long long)__ldg(s) - (i > 0 ? (unsigned long long)__ldg(s - 1) : 0ull);
                            }
                        }
                }
            }
            if (OUTLINE) {
                // counts of pixels i .. i + 3 of row r (those up to last)
                auto counts = [&](int i, int last, int r, uint32_t (&v)[4]) {
                    if (a.tier_code) {
                        const int j = jb + r;
                        const size_t b0 = (size_t)t * a.tier_bw * a.tier_bh + (size_t)(j >> 4) * a.tier_bw;
                        uint32_t code[4];
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) code[u] = i + u <= last ? __ldg(a.tier_code + b0 + ((i + u) >> 4)) : 0u;
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            v[u] = 0u;
                            if (i + u > last) continue;
                            if (!(code[u] & kTierMixed) || code[u] >= kTierMulti)
                                atomicOr(a.err, 4);   // never: such blocks are made mixed
                            else
                                v[u] = __ldg(a.tier_pcnt + (size_t)(code[u] & ~kTierMixed) * 256 + (j & 15) * 16 + ((i + u) & 15));
                        }
                    } else {
                        C w[5];
                        #pragma unroll
                        for (int u = 0; u < 5; ++u) w[u] = i + u - 1 <= last ? prefix_at(r, i + u) : C(0);
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = i + u <= last ? (uint32_t)(w[u + 1] - w[u]) : 0u;
                    }
                };
                OutlineQueue& Q = s_queue[OUTLINE ? warp : 0];
                int qn = 0;
                // the clip of the last 32 (or fewer) queued pixels
                auto drain = [&]() {
                    const int first = max(qn - 32, 0), x = first + lane;
                    if (x < qn) {
                        const int k = Q.k[x], i = (int)(Q.at[x] & 0xFFFFu), r = (int)(Q.at[x] >> 16), j = jb + r;
                        const uint32_t val = Q.val[x];
                        const float2 P0 = pf[k], P1 = pf[(k + 1 == n) ? 0 : k + 1];
                        bool ok = true;
                        if (a.line_filter) {
                            // varying interpolation along the line (projection of
                            // the pixel centre), kept within 0.5 px: line-bound.frag:221
                            const float cxp = (float)i + 0.5f, cyp = (float)j + 0.5f;
                            const float dx = __fsub_rn(P1.x, P0.x), dy = __fsub_rn(P1.y, P0.y);
                            const float l2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
                            ok = l2 > 0.0f;
                            const float tt = __fdiv_rn(__fadd_rn(__fmul_rn(__fsub_rn(cxp, P0.x), dx),
                                                                 __fmul_rn(__fsub_rn(cyp, P0.y), dy)), l2);
                            const float qx = __fadd_rn(P0.x, __fmul_rn(tt, dx));
                            const float qy = __fadd_rn(P0.y, __fmul_rn(tt, dy));
                            if (fabsf(__fsub_rn(qx, cxp)) >= 0.5f || fabsf(__fsub_rn(qy, cyp)) >= 0.5f) ok = false;
                        }
                        float frac;
                        if (ok && compute_fraction(P0.x, P0.y, P1.x, P1.y, (float)i, (float)j, (float)(i + 1), (float)(j + 1),
                                                   frac)) {
                            // inside test of the pixel centre: the coverage rule (an
                            // odd number of the row's crossings right of i)
                            bool inside = false;
                            if (r >= cl && r <= ch) {
                                if (slow) inside = inside_slow(i, r);
                                else
                                    for (int c = S.start[r] - base, e = c + S.cur[r]; c < e; ++c)
                                        inside ^= (int)(S.cross[c] & kColMask) > i;
                            }
                            if (frac > 0.5f) frac = __fsub_rn(1.0f, frac);
                            const int add = (int)ceilf(__fmul_rn(frac, (float)val));
                            if (inside) { b_fp += add; b_fp1 += val; }
                            else        { b_fn += add; b_fn1 += val; }
                        }
                    }
                    qn = first;
                    __syncwarp();
                };
                // (edge, row) pairs whose rectangles can touch: rows j with
                // j <= the edge's top and j + 1 >= its bottom
                spread_rows(
                    ne, lane, 0,
                    [&](int e, int& k, int& r0, int& cnt) {
                        k = overflow ? e : S.eidx[e];
                        const float2 P0 = pf[k], P1 = pf[(k + 1 == n) ? 0 : k + 1];
                        const float lo = fminf(P0.y, P1.y) - (float)(jb + 1), hi = fmaxf(P0.y, P1.y) - (float)jb;
                        r0 = max(lo > -32.0f ? (lo < 32.0f ? (int)ceilf(lo) : 32) : -32, ra);
                        cnt = max(min(hi < 32.0f ? (hi > -32.0f ? (int)floorf(hi) : -32) : 32, rb - 1) - r0 + 1, 0);
                    },
                    [](int k, int lo) { return __shfl_sync(0xffffffffu, k, lo); },
                    [&](bool live, int k, int r) {
                        int i0 = 0, i1 = -1;
                        if (live) {
                            const float2 P0 = pf[k], P1 = pf[(k + 1 == n) ? 0 : k + 1];
                            const float ylo = (float)(jb + r), yhi = (float)(jb + r + 1);
                            // x range of the edge inside the row and a pixel more on
                            // each side: on a nearly horizontal edge the clip's fp32
                            // rounding of y moves its ends by up to a pixel
                            float xa, xb;
                            if (P0.y == P1.y) {
                                xa = fminf(P0.x, P1.x);
                                xb = fmaxf(P0.x, P1.x);
                            } else {
                                const float ta = fminf(fmaxf((ylo - P0.y) / (P1.y - P0.y), 0.0f), 1.0f);
                                const float tb = fminf(fmaxf((yhi - P0.y) / (P1.y - P0.y), 0.0f), 1.0f);
                                const float x_a = P0.x + (P1.x - P0.x) * ta, x_b = P0.x + (P1.x - P0.x) * tb;
                                xa = fminf(x_a, x_b);
                                xb = fmaxf(x_a, x_b);
                            }
                            i0 = max((int)floorf(xa) - 1, 0);
                            i1 = min((int)floorf(xb) + 1, a.resx - 1);
                        }
                        // rounds of four pixels a lane: wide pairs one after the
                        // other, by the whole warp, then every lane its own (one
                        // place for the reads, the queue and the clip: inlined
                        // twice over, the code outgrew the instruction cache)
                        unsigned wide = __ballot_sync(FULL, i1 - i0 >= 16);
                        if ((wide >> lane) & 1u) i1 = -1 - i1;   // (kept for the others to read)
                        int wi = 0;
                        for (;;) {
                            int rk = k, rr = r, ri = i0, re = i1;
                            if (wide) {
                                const int src = __ffs(wide) - 1;
                                rk = __shfl_sync(FULL, k, src);
                                rr = __shfl_sync(FULL, r, src);
                                re = -1 - __shfl_sync(FULL, i1, src);
                                ri = __shfl_sync(FULL, i0, src) + wi + lane * 4;
                                wi += 128;
                                if (ri - lane * 4 + 128 > re) {
                                    wide &= wide - 1u;
                                    wi = 0;
                                }
                            } else {
                                if (!__any_sync(FULL, i0 <= i1)) break;
                                i0 += 4;
                            }
                            uint32_t v[4] = {0u, 0u, 0u, 0u};
                            if (ri <= re) counts(ri, re, rr, v);
                            #pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const unsigned m = __ballot_sync(FULL, v[u] != 0u);
                                if (v[u]) {
                                    const int x = qn + __popc(m & ((1u << lane) - 1u));
                                    Q.k[x] = rk;
                                    Q.at[x] = (uint32_t)(ri + u) | ((uint32_t)rr << 16);
                                    Q.val[x] = v[u];
                                }
                                qn += __popc(m);
                            }
                            __syncwarp();
                            #pragma unroll 1
                            while (qn >= 32) drain();
                        }
                    });
                if (qn > 0) drain();
            }
            __syncwarp();
            ra = rb;
        }
        if (SPANS) {
            acc_c = warp_sum_u64(acc_c);
            if (lane == 0 && acc_c) atomicAdd(a.out_count + p, acc_c);
            if (a.canvas_s) {
                acc_s = warp_sum_u64(acc_s);
                if (lane == 0 && acc_s) atomicAdd(a.out_sum + p, acc_s);
            }
        }
        if (OUTLINE) {
            b_fn = (long long)warp_sum_u64((unsigned long long)b_fn);
            b_fp = (long long)warp_sum_u64((unsigned long long)b_fp);
            b_fn1 = (long long)warp_sum_u64((unsigned long long)b_fn1);
            b_fp1 = (long long)warp_sum_u64((unsigned long long)b_fp1);
            if (lane == 0) {
                if (b_fn) atomicAdd((unsigned long long*)(a.out_bounds + p), (unsigned long long)b_fn);
                if (b_fp) atomicAdd((unsigned long long*)(a.out_bounds + a.P + p), (unsigned long long)b_fp);
                if (b_fn1) atomicAdd((unsigned long long*)(a.out_bounds + 2 * a.P + p), (unsigned long long)b_fn1);
                if (b_fp1) atomicAdd((unsigned long long*)(a.out_bounds + 3 * a.P + p), (unsigned long long)b_fp1);
            }
        }
    }
}

}  // namespace

void launch_row_prefix(uint32_t* counts, unsigned long long* wide, long long* sums, int resx, size_t rows, int sms,
                       cudaStream_t st) {
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>(rows, (size_t)sms * 8));
    k_row_prefix<<<blocks, kPrefixThreads, 0, st>>>(counts, wide, reinterpret_cast<unsigned long long*>(sums), resx, (int)rows);
    ++g_kernel_launches;
}

void launch_poly_bands(bool spans, bool outline, const PolyPassArgs& a, int sms, cudaStream_t st) {
    auto go = [&](auto kernel, auto prefix) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBW * 32, 0);
        kernel<<<sms * std::max(per_sm, 1), kBW * 32, 0, st>>>(a, prefix);
    };
    const bool w = a.canvas_w != nullptr;
    if (spans && outline) w ? go(k_poly_bands<true, true, unsigned long long>, a.canvas_w) : go(k_poly_bands<true, true, uint32_t>, a.canvas_c);
    else if (spans) w ? go(k_poly_bands<true, false, unsigned long long>, a.canvas_w) : go(k_poly_bands<true, false, uint32_t>, a.canvas_c);
    else go(k_poly_bands<false, true, uint32_t>, a.canvas_c);
    ++g_kernel_launches;
}

}  // namespace rj
