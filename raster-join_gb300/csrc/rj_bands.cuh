// rj_bands.cuh -- (edge, row) pairs of a band of pixel rows spread over a
// warp's lanes (the polygon-side passes over outlines).
#pragma once
#include "rj_device.cuh"

namespace rj {

constexpr int kBand = 16;          // pixel rows per work item

// Rows [r0, r1] of the band (relative to jb) whose centre line the edge
// with fixed-point ends y = ay, by crosses: ylo < cy <= yhi, cy = j * 256 + 128.
__device__ __forceinline__ void edge_rows(int32_t ay, int32_t by, int jb, int& r0, int& r1) {
    const int64_t ylo = min(ay, by), yhi = max(ay, by);
    const int64_t a0 = ((ylo - kSub / 2) >> kSubpixelBits) + 1 - jb;
    const int64_t a1 = ((yhi - kSub / 2) >> kSubpixelBits) - jb;
    r0 = (int)(a0 < 0 ? 0 : a0);
    r1 = (int)(a1 > kBand - 1 ? kBand - 1 : a1);
}

// f(q, r) for every row r of the ranges that range(e, q, r0, cnt) gives the
// items e < ne (rows r0 .. r0 + cnt - 1, payload q), spread over the lanes: an
// edge of 16 rows gives 16 lanes work instead of one lane 16 rounds.  Every
// lane calls this (warp-uniform loops).
template <class Q, class R, class S, class F>
__device__ __forceinline__ void spread_rows(int ne, int lane, Q q, R&& range, S&& shuffle, F&& f) {
    const unsigned FULL = 0xffffffffu;
    for (int e0 = 0; e0 < ne; e0 += 32) {
        const int e = e0 + lane;
        int r0 = 0, cnt = 0;
        if (e < ne) range(e, q, r0, cnt);
        int incl = cnt;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(FULL, incl, 31);
        for (int base = 0; base < total; base += 32) {
            const int idx = base + lane;
            int lo = 0, hi = 31;   // the first lane whose inclusive count exceeds idx
            #pragma unroll
            for (int s = 0; s < 5; ++s) {
                const int mid = (lo + hi) >> 1;
                if (__shfl_sync(FULL, incl, mid) > idx) hi = mid; else lo = mid + 1;
            }
            const Q qe = shuffle(q, lo);
            const int r = __shfl_sync(FULL, r0, lo) + idx - (__shfl_sync(FULL, incl, lo) - __shfl_sync(FULL, cnt, lo));
            f(idx < total, qe, r);
        }
    }
}

// f(q, r) for every (edge, band row) pair whose row centre line the edge's
// y range spans; edge(e) returns staged edge e < ne.
template <class E, class F>
__device__ __forceinline__ void for_edge_rows(int ne, int jb, int lane, E&& edge, F&& f) {
    spread_rows(
        ne, lane, make_int4(0, 0, 0, 0),
        [&](int e, int4& q, int& r0, int& cnt) {
            q = edge(e);
            int r1;
            edge_rows(q.y, q.w, jb, r0, r1);
            cnt = max(r1 - r0 + 1, 0);
        },
        [](const int4& q, int lo) {
            return make_int4(__shfl_sync(0xffffffffu, q.x, lo), __shfl_sync(0xffffffffu, q.y, lo),
                             __shfl_sync(0xffffffffu, q.z, lo), __shfl_sync(0xffffffffu, q.w, lo));
        },
        [&](bool live, const int4& q, int r) {
            if (live) f(q, r);
        });
}

}  // namespace rj
