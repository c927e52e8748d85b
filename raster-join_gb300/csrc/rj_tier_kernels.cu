// rj_tier_kernels.cu -- tiered canvas for fine resolutions.
//
// A raster canvas of 10^8-10^9 pixels is mostly the interiors of polygons.
// The tiered canvas keeps it as 16 x 16-pixel blocks:
//   * a block every pixel centre of which lies inside one polygon ("full")
//     is one entry: the polygon id (label form) or one count / sum (canvas
//     form);
//   * a block no polygon reaches is empty;
//   * only "mixed" blocks (crossed by an edge, or full for one polygon and
//     touched by another) keep per-pixel data, in a compact slot of 256
//     pixels.
// Coverage is the same pixel-centre rule as the flat canvas (exact integer
// crossings of the row centre lines; a pixel is inside when an odd number of
// crossings lie at or left of it), so every result is identical; the work
// becomes proportional to polygon perimeters and mixed blocks instead of
// polygon areas.
//
// One warp per (tile, polygon, band of 16 rows); bands are aligned to block
// rows.  The work of a band is proportional to the crossings of its rows and
// to the blocks the polygon's outline passes through (plus one entry per full
// block), not to the pixels of its area:
//   * the band's (edge, row) crossing pairs are spread over the lanes, one
//     exact crossing each;
//   * sweep 1 -- every crossing of a live row toggles one bit of a per-row
//     block bitmap (at the first block whose first pixel lies at or right of
//     it) and, when it falls strictly inside a block, flags that block; a
//     prefix XOR over the bitmap gives each block's coverage at its first
//     pixel, which holds for the whole block row unless the block is flagged.
//     Over the 16 rows: I = blocks covered throughout (full for the polygon),
//     U = blocks the polygon covers somewhere.
//   * the blocks whose pixels matter (U and mixed; a mixed block's points are
//     in its pixel slot only) are listed, up to 64 at a time; sweep 2 toggles per-pixel bits of
//     the listed blocks only, and their 16-bit row masks follow from the
//     block's first-pixel coverage and a 16-bit prefix XOR;
//   * the listed blocks' pixel slots are then read or written by the whole
//     warp, eight pixels a lane with vector loads and stores.
//
// Measured (2,000 stars at 1 m, 40,000 x 40,000 pixels): CLASSIFY 0.83 ms and
// REDUCE 2.35, before the crossings did without 64-bit divisions and bands
// without dependent loads 1.43 and 2.78.  A launch of 30 polygons is 1.9
// instructions per cycle and SM with a third of the warps resident (54 KB of
// shared memory per block): issue, latency and the last bands share the time.
#include "rj_bands.cuh"
#include "rj_launch.h"
#include "rj_point_map.cuh"

namespace rj {

namespace {

constexpr int kTW = 8;            // warps per block
constexpr int kTBand = kBand;     // rows per work item: one block row
// Staged edges per warp.  Where a band has more, up to four times as many are
// staged as vertex numbers and read from global memory; where it has more than
// that, every sweep stages them anew, so many at a time.  (Going through all of
// the polygon's edges instead, four rings of 160,000 vertices on 20,000 x 20,000
// pixels, counts: 26.6 ms from 113 edges on, 13.6 from 257 on; now 8.1.  Shared
// memory for 256 edges leaves three blocks per SM instead of four.)
constexpr int kTEdgeCap = 112;
constexpr int kTIndexCap = kTEdgeCap * (int)(sizeof(int4) / sizeof(int));
constexpr int kTBW = 16;          // block-bitmap words per row: 512 block columns = 8192 pixels
constexpr int kTList = 64;        // blocks whose pixels one round visits

// Per-warp shared memory.  X, C and M are zero between work items.
struct TierWarp {
    int4 edge[kTEdgeCap];               // staged edges of the band
    uint32_t X[kTBand * kTBW];          // block toggles, then coverage at each block's first pixel
    uint32_t C[kTBand * kTBW];          // blocks with a crossing inside (pixel offsets 1..15)
    uint32_t M[kTList * kTBand / 2];    // listed blocks: pixel toggles, then row masks (two rows a word)
    uint32_t slot[kTList];              // listed blocks' slots
    uint16_t list[kTList];              // listed block columns (relative to bc_lo)
    uint8_t map[kTBW * 32];             // block column -> list index, 0xFF when not listed
};
static_assert(sizeof(TierWarp) % 16 == 0, "TierWarp keeps 16-byte alignment");
constexpr size_t kTierSmem = (size_t)kTW * sizeof(TierWarp);

__device__ __forceinline__ bool tier_mixed(uint32_t code) { return code >= kTierMixed && code < kTierMulti; }

// bits [a, b) of a word, 0 <= a < b <= 32
__device__ __forceinline__ uint32_t bitrange(int a, int b) {
    return (b >= 32 ? 0xFFFFFFFFu : ((1u << b) - 1u)) & ~((1u << a) - 1u);
}
// inclusive prefix parity: bit k = XOR of bits 0..k
__device__ __forceinline__ uint32_t prefix_xor(uint32_t x) {
    x ^= x << 1;
    x ^= x << 2;
    x ^= x << 4;
    x ^= x << 8;
    x ^= x << 16;
    return x;
}

// The numbers of the edges' vertices, staged from k0 on; returns how many there
// are and the vertex reached.  (A call, as few bands come here: inlined for
// every sweep it cost 1B points at 1 m 6 to 10 us of 2513, so 2 to 6.)
__device__ __noinline__ int2 stage_numbers(const int2* __restrict__ pv, int n, int64_t lo, int64_t hi, int k0, int room, int* index) {
    const int m = stage_edges(pv, n, lo, hi, (int)(threadIdx.x & 31u), k0, room, [&](int pos, int k, const int4&) { index[pos] = k; });
    __syncwarp();
    return make_int2(m, k0);
}

template <int MODE>
__global__ void __launch_bounds__(kTW * 32, 4) k_tier_pass(PolyPassArgs a, TierArgs tr) {
    extern __shared__ int4 s_tier[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    const int TP = a.T * a.P;
    TierWarp& S = reinterpret_cast<TierWarp*>(s_tier)[warp];
    BandItems work(a.band_start, TP, a.work_ctr, kTW, warp, lane);
    for (int w = lane; w < kTBand * kTBW; w += 32) {
        S.X[w] = 0u;
        S.C[w] = 0u;
    }
    for (int w = lane; w < kTList * kTBand / 2; w += 32) S.M[w] = 0u;
    __syncwarp();
    const int hw = lane & 15, half = lane >> 4;   // sweep 1: row 2k + half, block word hw
    for (;;) {
        const int item = work.take(a.band_start, TP, a.work_ctr, lane);
        if (item < 0) break;
        const int tp = work.tp;
        const int t = tp / a.P, p = tp - t * a.P;
        const int band = item - work.tp_first;
        const int4 ia = a.info_a[tp];
        const int2 ib = a.info_b[tp];
        const int i_lo = ia.x, i_hi = ia.y, j_lo = ib.x, j_hi = ib.y;
        const int jb = ia.z + band * kTBand;            // a multiple of 16
        const int br = jb >> 4;
        const int v0 = __ldg(a.pindex + p);
        const int n = __ldg(a.pindex + p + 1) - v0;
        const int2* pv = a.wv + (size_t)t * a.V + v0;
        const size_t blk0 = (size_t)t * tr.bw * tr.bh + (size_t)br * tr.bw;
        const int bc_lo = i_lo >> 4;
        const int nbc = (i_hi >> 4) - bc_lo + 1;        // block columns of the range (<= 512)
        if (nbc > kTBW * 32) continue;                  // never: resx <= 8192

        // stage the edges that can cross a row centre of the band
        const int64_t band_lo = (int64_t)jb * kSub - kSub;
        const int64_t band_hi = (int64_t)(jb + kTBand) * kSub + kSub;
        int* index = reinterpret_cast<int*>(S.edge);
        const int nb = stage_edges(pv, n, band_lo, band_hi, lane, [&](int pos, int, const int4& e) {
            if (pos < kTEdgeCap) S.edge[pos] = e;
        });
        const bool numbers = nb > kTEdgeCap, pieces = nb > kTIndexCap;
        __syncwarp();
        if (numbers && !pieces) stage_numbers(pv, n, band_lo, band_hi, 0, INT_MAX, index);
        auto edge_at = [&](int e) -> int4 {
            if (!numbers) return S.edge[e];
            const int k = index[e];
            const int2 A = pv[k];
            const int2 B = pv[(k + 1 == n) ? 0 : k + 1];
            return make_int4(A.x, A.y, B.x, B.y);
        };
        // f(number of staged edges) until the band's edges are through
        auto for_staged = [&](auto&& f) {
            for (int k = pieces ? 0 : n, m = nb;;) {
                if (pieces) {
                    const int2 s = stage_numbers(pv, n, band_lo, band_hi, k, kTIndexCap, index);
                    m = s.x;
                    k = s.y;
                }
                f(m);
                __syncwarp();
                if (k >= n) break;
            }
        };
        if (MODE == MODE_TIER_CLASSIFY && tr.outline) {
            // blocks within two pixels of an edge near this band (rows
            // jb - 2 .. jb + 17) become mixed: the error-bound outline pass
            // reads per-pixel counts up to a pixel beside each edge, rows one
            // beyond the polygon's included
            const float ylo = (float)(jb - 2), yhi = (float)(jb + kTBand + 2);
            for_staged([&](int ne) {
                for (int e = lane; e < ne; e += 32) {
                    const int4 q = edge_at(e);
                    const float ax = q.x * (1.0f / kSub), ay = q.y * (1.0f / kSub);
                    const float bx = q.z * (1.0f / kSub), by = q.w * (1.0f / kSub);
                    const float y0 = fmaxf(fminf(ay, by), ylo), y1 = fminf(fmaxf(ay, by), yhi);
                    if (!(y0 <= y1)) continue;
                    float x0, x1;
                    if (ay == by) {
                        x0 = fminf(ax, bx);
                        x1 = fmaxf(ax, bx);
                    } else {
                        const float ta = fminf(fmaxf((y0 - ay) / (by - ay), 0.0f), 1.0f);
                        const float tb = fminf(fmaxf((y1 - ay) / (by - ay), 0.0f), 1.0f);
                        const float xa = ax + (bx - ax) * ta, xb = ax + (bx - ax) * tb;
                        x0 = fminf(xa, xb);
                        x1 = fmaxf(xa, xb);
                    }
                    const int c0 = max((int)floorf(x0) - 2, 0), c1 = min((int)floorf(x1) + 2, a.resx - 1);
                    const int r0 = max((int)floorf(y0) - 2, 0), r1 = min((int)floorf(y1) + 2, a.resy - 1);
                    if (c0 > c1 || r0 > r1) continue;
                    const size_t tile0 = (size_t)t * tr.bw * tr.bh;
                    for (int br2 = r0 >> 4; br2 <= (r1 >> 4); ++br2)
                        for (int bc = c0 >> 4; bc <= (c1 >> 4); ++bc) tr.mixed[tile0 + (size_t)br2 * tr.bw + bc] = 1u;
                }
            });
        }

        if (nbc <= 0) continue;                         // outline rows only

        // rows of the band inside the polygon's crossing rows and the canvas
        const int rl = max(j_lo, jb) - jb, rh = min(min(j_hi, a.resy - 1), jb + kTBand - 1) - jb;
        const uint32_t live = rl <= rh ? bitrange(rl, rh + 1) : 0u;
        if (!live) continue;

        // sweep 1: block toggles and inside-crossing flags per live row
        for_staged([&](int ne) {
            for_edge_rows(ne, jb, lane, edge_at, [&](const int4& q, int r) {
                const int32_t cy = (jb + r) * kSub + kSub / 2;
                if (!((live >> r) & 1u) || !cross_row(q.y, q.w, cy)) return;
                const int L = max(cross_L(q.x, q.y, q.z, q.w, cy), i_lo);
                if (L > i_hi) return;
                const int rb = ((L + 15) >> 4) - bc_lo;
                if (rb < nbc) atomicXor(&S.X[r * kTBW + (rb >> 5)], 1u << (rb & 31));
                if (L & 15) {
                    const int cb = (L >> 4) - bc_lo;
                    atomicOr(&S.C[r * kTBW + (cb >> 5)], 1u << (cb & 31));
                }
            });
        });
        // block columns [fb, lb] lie wholly inside [i_lo, i_hi]; word hw's valid blocks
        const int fb = ((i_lo + 15) >> 4) - bc_lo, lb = ((i_hi + 1) >> 4) - 1 - bc_lo;
        const int wa = max(fb - hw * 32, 0), wb = min(lb - hw * 32 + 1, 32);
        const int va = min(nbc - hw * 32, 32);
        const uint32_t valid = va > 0 ? bitrange(0, va) : 0u;
        uint32_t I = (live == 0xFFFFu && wa < wb) ? bitrange(wa, wb) : 0u, U = 0u;
        #pragma unroll 2
        for (int r2 = 0; r2 < kTBand; r2 += 2) {
            const int r = r2 + half;
            const int idx = r * kTBW + hw;
            const uint32_t tg = S.X[idx], c = S.C[idx];
            uint32_t x = prefix_xor(tg);
            const unsigned odd = __ballot_sync(FULL, (__popc(tg) & 1) != 0);
            if (__popc((odd >> (half * 16)) & ((1u << hw) - 1u)) & 1) x = ~x;
            S.X[idx] = x;
            S.C[idx] = 0u;
            if ((live >> r) & 1u) {
                I &= x & ~c;
                U |= (x | c) & valid;
            }
        }
        I &= __shfl_xor_sync(FULL, I, 16);
        U |= __shfl_xor_sync(FULL, U, 16);
        const int nbw = (nbc + 31) >> 5;

        if (MODE == MODE_TIER_CLASSIFY) {
            // block columns: full for p, or touched (mixed)
            for (int k = 0; k < nbw; ++k) {
                const uint32_t Iw = __shfl_sync(FULL, I, k), Uw = __shfl_sync(FULL, U, k);
                if (!Uw) continue;
                const int rel = k * 32 + lane;
                if (!((Uw >> lane) & 1u)) continue;
                const size_t b = blk0 + bc_lo + rel;
                if ((Iw >> lane) & 1u) {
                    atomicAdd(tr.full + b, (1ull << 32) + (unsigned long long)p);
                } else {
                    tr.mixed[b] = 1u;
                }
            }
            for (int w = lane; w < kTBand * kTBW; w += 32) S.X[w] = 0u;
            __syncwarp();
            continue;
        }

        unsigned long long acc_c = 0;
        long long acc_s = 0;
        // listed blocks: covered and mixed (a block covered but not full is
        // mixed; reduce: the full blocks that are not mixed give their totals)
        uint32_t Lw = 0u;   // lane k < nbw: listed blocks of word k
        // (the words' block codes are loaded four words at a time)
        for (int k0 = 0; k0 < nbw; k0 += 4) {
            uint32_t code[4], cb[4];
            long long sb[4];
            #pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t Uw = k0 + u < nbw ? __shfl_sync(FULL, U, k0 + u) : 0u;
                code[u] = (Uw >> lane) & 1u ? __ldg(tr.code + blk0 + bc_lo + (k0 + u) * 32 + lane) : kTierEmpty;
            }
            if (MODE == MODE_TIER_REDUCE) {
                #pragma unroll
                for (int u = 0; u < 4; ++u) {
                    // a covered block that is not mixed is full: its total
                    const bool whole = code[u] != kTierEmpty && !tier_mixed(code[u]);
                    const size_t b = blk0 + bc_lo + (k0 + u) * 32 + lane;
                    cb[u] = whole ? __ldg(tr.bcnt + b) : 0u;
                    sb[u] = whole && tr.bsum ? __ldg(tr.bsum + b) : 0;
                }
                #pragma unroll
                for (int u = 0; u < 4; ++u) {
                    acc_c += cb[u];
                    acc_s += sb[u];
                }
            }
            #pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t m = __ballot_sync(FULL, tier_mixed(code[u]));
                if (lane == k0 + u) Lw = m;
            }
        }
        // list positions: exclusive prefix of the words' counts
        const int cnt = lane < nbw ? __popc(Lw) : 0;
        int pre = cnt;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, pre, o);
            if (lane >= o) pre += v;
        }
        const int nlist = __shfl_sync(FULL, pre, 31);
        pre -= cnt;
        for (int start = 0; start < nlist; start += kTList) {
            const int nk = min(kTList, nlist - start);
            for (int w = lane; w < kTBW * 32 / 4; w += 32) reinterpret_cast<uint32_t*>(S.map)[w] = 0xFFFFFFFFu;
            __syncwarp();
            if (lane < nbw && pre < start + nk && pre + cnt > start) {
                uint32_t m = Lw;
                int g = pre;
                while (m && g < start + nk) {
                    const int bit = __ffs(m) - 1;
                    m &= m - 1u;
                    if (g >= start) {
                        S.map[lane * 32 + bit] = (uint8_t)(g - start);
                        S.list[g - start] = (uint16_t)(lane * 32 + bit);
                        S.slot[g - start] = __ldg(tr.code + blk0 + bc_lo + lane * 32 + bit) & ~kTierMixed;
                    }
                    ++g;
                }
            }
            __syncwarp();
            // sweep 2: pixel toggles of the listed blocks (crossings inside a
            // block only; one at a block's first pixel is in X already)
            for_staged([&](int ne) {
                for_edge_rows(ne, jb, lane, edge_at, [&](const int4& q, int r) {
                    const int32_t cy = (jb + r) * kSub + kSub / 2;
                    if (!((live >> r) & 1u) || !cross_row(q.y, q.w, cy)) return;
                    const int L = max(cross_L(q.x, q.y, q.z, q.w, cy), i_lo);
                    if (L > i_hi || !(L & 15)) return;
                    const int k = S.map[(L >> 4) - bc_lo];
                    if (k != 0xFF) atomicXor(&S.M[k * 8 + (r >> 1)], (1u << (L & 15)) << ((r & 1) * 16));
                });
            });
            // row masks: coverage at the block's first pixel, then the block's
            // own crossings, clipped to [i_lo, i_hi]
            for (int w = lane; w < nk * 8; w += 32) {
                const int k = w >> 3, rp = (w & 7) * 2;
                const int rel = S.list[k];
                const int x0 = (bc_lo + rel) * 16;
                const int ka = max(i_lo - x0, 0), kb = min(i_hi - x0, 15);
                const uint32_t rng = bitrange(ka, kb + 1);
                const uint32_t tg = S.M[w];
                uint32_t out = 0u;
                #pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = rp + h;
                    if (!((live >> r) & 1u)) continue;
                    uint32_t x = prefix_xor((tg >> (h * 16)) & 0xFFFFu) & 0xFFFFu;
                    if ((S.X[r * kTBW + (rel >> 5)] >> (rel & 31)) & 1u) x ^= 0xFFFFu;
                    out |= (x & rng) << (h * 16);
                }
                S.M[w] = out;
            }
            __syncwarp();
            // the listed blocks' pixels: lane = (row, half row of 8 pixels)
            const int pr = lane >> 1, ph = (lane & 1) * 8;
            #pragma unroll 4
            for (int k = 0; k < nk; ++k) {
                const uint32_t m8 = (S.M[k * 8 + (pr >> 1)] >> ((pr & 1) * 16 + ph)) & 0xFFu;
                if (!m8) continue;
                const size_t q = (size_t)S.slot[k] * 256 + (size_t)pr * 16 + ph;
                if (MODE == MODE_TIER_LABEL) {
                    uint16_t* dst = tr.plabel + q;
                    if (m8 == 0xFFu) {
                        const uint32_t pp = (uint32_t)p | ((uint32_t)p << 16);
                        *reinterpret_cast<uint4*>(dst) = make_uint4(pp, pp, pp, pp);
                    } else {
                        #pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if ((m8 >> i) & 1u) dst[i] = (uint16_t)p;
                    }
                    acc_c += (unsigned)__popc(m8);
                } else {
                    const uint4 c0 = __ldg(reinterpret_cast<const uint4*>(tr.pcnt + q));
                    const uint4 c1 = __ldg(reinterpret_cast<const uint4*>(tr.pcnt + q + 4));
                    acc_c += (unsigned long long)((m8 & 1u) ? c0.x : 0u) + ((m8 & 2u) ? c0.y : 0u) +
                             ((m8 & 4u) ? c0.z : 0u) + ((m8 & 8u) ? c0.w : 0u) + ((m8 & 16u) ? c1.x : 0u) +
                             ((m8 & 32u) ? c1.y : 0u) + ((m8 & 64u) ? c1.z : 0u) + ((m8 & 128u) ? c1.w : 0u);
                    if (tr.psum) {
                        const longlong2* ps = reinterpret_cast<const longlong2*>(tr.psum + q);
                        #pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const longlong2 v = __ldg(ps + i);
                            if ((m8 >> (2 * i)) & 1u) acc_s += v.x;
                            if ((m8 >> (2 * i + 1)) & 1u) acc_s += v.y;
                        }
                    }
                }
            }
            __syncwarp();   // every lane has read its masks
            for (int w = lane; w < nk * 8; w += 32) S.M[w] = 0u;
            __syncwarp();
        }
        for (int w = lane; w < kTBand * kTBW; w += 32) S.X[w] = 0u;
        __syncwarp();
        acc_c = warp_sum_u64(acc_c);
        if (MODE == MODE_TIER_LABEL) {
            if (lane == 0 && acc_c) atomicAdd(a.covered, acc_c);
        } else {
            if (tr.bsum || tr.psum) acc_s = (long long)warp_sum_u64((unsigned long long)acc_s);
            if (lane == 0 && acc_c) atomicAdd(a.out_count + p, acc_c);
            if (lane == 0 && acc_s != 0) atomicAdd(a.out_sum + p, (unsigned long long)acc_s);
        }
    }
}

// code[b]: kTierMixed | slot for mixed blocks, else the full polygon (or
// empty / multi); counts the multi blocks (two polygons cover them whole).
// Slots are handed out by one atomic per 256 blocks (their order does not
// matter; one per warp took 150 us for 6.2M blocks, this 35), or each block is
// its own slot, whose pixel labels this then clears, a warp writing one
// block's 512 bytes at a time.
constexpr int kCodeThreads = 256;
__global__ void __launch_bounds__(kCodeThreads) k_tier_codes(TierArgs tr, size_t nblk, unsigned long long* multi, int* err) {
    __shared__ uint32_t s_warp[kCodeThreads / 32];
    __shared__ uint32_t s_base;
    unsigned long long c = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 none = make_uint4(~0u, ~0u, ~0u, ~0u);
    // (block-uniform trip count)
    for (size_t first = (size_t)blockIdx.x * kCodeThreads; first < nblk; first += (size_t)gridDim.x * kCodeThreads) {
        const size_t b = first + threadIdx.x, b0 = b - lane;
        const bool mixed = b < nblk && tr.mixed[b] != 0u;
        const unsigned m = __ballot_sync(0xffffffffu, mixed);
        uint32_t slot = (uint32_t)b;
        if (!tr.own_place) {
            if (lane == 0) s_warp[warp] = (uint32_t)__popc(m);
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t n = 0;
                #pragma unroll
                for (int w = 0; w < kCodeThreads / 32; ++w) {
                    const uint32_t k = s_warp[w];
                    s_warp[w] = n;
                    n += k;
                }
                s_base = n ? atomicAdd(tr.nslots, n) : 0u;
            }
            __syncthreads();
            slot = s_base + s_warp[warp] + __popc(m & ((1u << lane) - 1u));
            __syncthreads();
        }
        if (b < nblk) {
            const unsigned long long f = tr.full[b];
            const uint32_t n = (uint32_t)(f >> 32);
            uint32_t code = mixed ? kTierMixed | slot : n == 0 ? kTierEmpty : n == 1 ? (uint32_t)f : kTierMulti;
            if (mixed && !tr.own_place && slot >= tr.cap) {   // (the host runs the query again with the exact number)
                atomicOr(err, kErrSlots);
                code = kTierEmpty;
            }
            tr.code[b] = code;
            c += n > 1;
        }
        if (tr.own_place)
            for (unsigned w = m; w; w &= w - 1u) reinterpret_cast<uint4*>(tr.plabel + (b0 + __ffs(w) - 1) * 256)[lane] = none;
    }
    c = warp_sum_u64(c);
    if (lane == 0 && c) atomicAdd(multi, c);
}

__global__ void k_tier_clear(TierArgs tr, size_t nblk) {
    const int lane = threadIdx.x & 31;
    const uint4 none = make_uint4(~0u, ~0u, ~0u, ~0u), zero = make_uint4(0u, 0u, 0u, 0u);
    for (size_t b0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) - lane; b0 < nblk;
         b0 += (size_t)gridDim.x * blockDim.x) {
        const size_t b = b0 + lane;
        const uint32_t code = b < nblk ? __ldg(tr.code + b) : kTierEmpty;
        if (b < nblk && tr.bcnt) tr.bcnt[b] = 0u;
        if (b < nblk && tr.bsum) tr.bsum[b] = 0;
        for (unsigned m = __ballot_sync(0xffffffffu, tier_mixed(code)); m; m &= m - 1u) {
            const size_t at = (size_t)(__shfl_sync(0xffffffffu, code, __ffs(m) - 1) & ~kTierMixed) * 256;
            if (tr.plabel) reinterpret_cast<uint4*>(tr.plabel + at)[lane] = none;
            if (tr.pcnt) {
                reinterpret_cast<uint4*>(tr.pcnt + at)[lane] = zero;
                reinterpret_cast<uint4*>(tr.pcnt + at)[lane + 32] = zero;
            }
            if (tr.psum)
                #pragma unroll
                for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(tr.psum + at)[lane + 32 * i] = zero;
        }
    }
}

// labelled pixels of the mixed blocks (overlap check: equals the pixel writes
// when no two polygons share a pixel centre), a warp per 32 blocks
__global__ void k_tier_nonempty(TierArgs tr, size_t nblk, unsigned long long* count) {
    unsigned long long c = 0;
    const int lane = threadIdx.x & 31;
    for (size_t b0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) - lane; b0 < nblk;
         b0 += (size_t)gridDim.x * blockDim.x) {
        const uint32_t code = b0 + lane < nblk ? __ldg(tr.code + b0 + lane) : kTierEmpty;
        for (unsigned m = __ballot_sync(0xffffffffu, tier_mixed(code)); m; m &= m - 1u) {
            const uint32_t slot = __shfl_sync(0xffffffffu, code, __ffs(m) - 1) & ~kTierMixed;
            const uint4 v = reinterpret_cast<const uint4*>(tr.plabel + (size_t)slot * 256)[lane];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            #pragma unroll
            for (int i = 0; i < 4; ++i) c += ((w[i] & 0xFFFFu) != kEmptyLabel) + ((w[i] >> 16) != kEmptyLabel);
        }
    }
    c = warp_sum_u64(c);
    if (lane == 0 && c) atomicAdd(count, c);
}

}  // namespace

size_t tier_smem_bytes() { return kTierSmem; }

void launch_tier_pass(int mode, const PolyPassArgs& a, const TierArgs& tr, int sms, cudaStream_t st) {
    ++g_kernel_launches;
    auto go = [&](auto kernel) {
        // every instance needs the opt-in (the three kernels share one pointer type)
        allow_smem(reinterpret_cast<const void*>(kernel), kTierSmem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTW * 32, kTierSmem);
        kernel<<<sms * std::max(per_sm, 1), kTW * 32, kTierSmem, st>>>(a, tr);
    };
    switch (mode) {
        case MODE_TIER_CLASSIFY: go(k_tier_pass<MODE_TIER_CLASSIFY>); break;
        case MODE_TIER_LABEL: go(k_tier_pass<MODE_TIER_LABEL>); break;
        default: go(k_tier_pass<MODE_TIER_REDUCE>); break;
    }
}

void launch_tier_codes(const TierArgs& tr, size_t nblk, unsigned long long* multi, int* err, int sms, cudaStream_t st) {
    const int blocks = (int)std::min<size_t>((nblk + 255) / 256, (size_t)sms * 16);
    k_tier_codes<<<std::max(blocks, 1), kCodeThreads, 0, st>>>(tr, nblk, multi, err);
    ++g_kernel_launches;
}

void launch_tier_clear(const TierArgs& tr, size_t nblk, int sms, cudaStream_t st) {
    const int blocks = (int)std::min<size_t>((nblk + 255) / 256, (size_t)sms * 16);
    k_tier_clear<<<std::max(blocks, 1), 256, 0, st>>>(tr, nblk);
    ++g_kernel_launches;
}

void launch_tier_nonempty(const TierArgs& tr, size_t nblk, unsigned long long* count, int sms, cudaStream_t st) {
    const int blocks = (int)std::min<size_t>((nblk + 255) / 256, (size_t)sms * 16);
    k_tier_nonempty<<<std::max(blocks, 1), 256, 0, st>>>(tr, nblk, count);
    ++g_kernel_launches;
}

}  // namespace rj
