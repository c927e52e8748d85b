// rj_bands.cuh -- (edge, row) pairs of a band of pixel rows spread over a
// warp's lanes (the polygon-side passes over outlines).
#pragma once
#include <climits>

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

// Work items (tile, polygon, band) of a persistent warp.  A pass over few items
// is latency from end to end, so every dependent load saved counts: up to two
// items a warp are dealt out (neighbours to different SMs), more are taken from
// the counter a few at a time, the next ones asked for before these are worked
// on; the owner is looked up when it changes.  Dealing them out took a count
// over 20,000 points and 64 cells at 100 m from 93 to 89 us, a prepared average
// over 1M points and 260 cells at 10 m from 92 to 86; with more items than that
// the counter's balance is worth its latency.
struct BandItems {
    int next, first, last, chunk, step, total;
    int tp, tp_first, tp_last;      // owner of the current item, its items [tp_first, tp_last)
    __device__ __forceinline__ BandItems(const int* band_start, int TP, unsigned* ctr, int warps, int warp, int lane) {
        total = band_start[TP];
        const int n = (int)gridDim.x * warps;
        step = total <= 2 * n ? n : 0;
        chunk = step ? 1 : min(max(total / (n * 4), 1), 4);
        next = step ? warp * (int)gridDim.x + (int)blockIdx.x : lane == 0 ? (int)atomicAdd(ctr, (unsigned)chunk) : 0;
        first = last = 0;
        tp = -1;
        tp_first = tp_last = 0;
    }
    // the next item, or -1 (the whole warp calls this)
    __device__ __forceinline__ int take(const int* band_start, int TP, unsigned* ctr, int lane) {
        if (first >= last) {
            first = step ? next : __shfl_sync(0xffffffffu, next, 0);
            if (first >= total) return -1;
            last = min(first + chunk, total);
            if (step) next += step;
            else if (lane == 0) next = (int)atomicAdd(ctr, (unsigned)chunk);
        }
        const int item = first++;
        if (tp < 0 || item >= tp_last) {
            tp = warp_find_owner(band_start, TP, item, lane);
            tp_first = __ldg(band_start + tp);
            tp_last = __ldg(band_start + tp + 1);
        }
        return item;
    }
};

// Edges of the ring pv[0, n) that meet the fixed-point rows [lo, hi], staged in
// order from vertex k0 on (f(position, vertex, edge) for each that is taken);
// returns how many there are.  Four rounds of vertices are loaded before the
// first is used; the last rounds are those after which there is no room for
// another four, and k0 is left behind them.
template <class F>
__device__ __forceinline__ int stage_edges(const int2* __restrict__ pv, int n, int64_t lo, int64_t hi, int lane, int& k0,
                                           int room, F&& f) {
    int nb = 0;
    for (; k0 < n && nb <= room - 128; k0 += 128) {
        int2 A[4], B[4];
        #pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * 32 + lane;
            A[u] = B[u] = make_int2(0, 0);
            if (k < n) {
                A[u] = pv[k];
                B[u] = pv[(k + 1 == n) ? 0 : k + 1];
            }
        }
        #pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * 32 + lane;
            const bool take = k < n && max(A[u].y, B[u].y) >= lo && min(A[u].y, B[u].y) <= hi;
            const unsigned m = __ballot_sync(0xffffffffu, take);
            if (take) f(nb + __popc(m & ((1u << lane) - 1u)), k, make_int4(A[u].x, A[u].y, B[u].x, B[u].y));
            nb += __popc(m);
        }
    }
    return nb;
}

template <class F>
__device__ __forceinline__ int stage_edges(const int2* __restrict__ pv, int n, int64_t lo, int64_t hi, int lane, F&& f) {
    int k0 = 0;
    return stage_edges(pv, n, lo, hi, lane, k0, INT_MAX, f);
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
