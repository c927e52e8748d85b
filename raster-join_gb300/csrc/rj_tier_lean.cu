// rj_tier_lean.cu -- lean point pass of the raster join over a tiered canvas
// in its canvas form (16 x 16-pixel blocks: one count / sum per full block,
// per-pixel counts in the slots of mixed blocks; rj_tier_kernels.cu), on one
// or several canvas tiles.  The counterpart of the generic pass's
// TierSplatMapper (rj_point_map.cuh) with the lean passes' structure:
// coalesced point-pair loads, interval-form filters, the exact snapped pixel
// (rj_lean.cuh), no warp grouping.
//
// Tiles: per axis the tile is guessed with one multiplication; when the
// pixel in the guessed tile lies far enough inside it (TileAxis::edge, one pixel
// unless the canvas is far from the origin), no other tile's window can hold the
// point and that is the only hit.  Otherwise (near a seam, or a guess off by one) the guessed tile and both
// neighbours are tried exactly, as the generic mapping does: near a seam a
// point can fall in two tiles' windows and counts in both (every tile is
// rendered with all points, RasterJoin.cpp:224-231).
//
// One count (and sum) per point with plain global atomics: into the pixel slot
// of a mixed block, else into the block's total (an empty block keeps
// nothing); the polygon pass reduces them.
#include "rj_label_core.cuh"

namespace rj {

namespace {

template <int NCOL>
__device__ __forceinline__ bool tl_pass(const LeanCols& lc, const uint32_t (&v)[NCOL > 0 ? NCOL : 1]) {
    bool ok = true;
    #pragma unroll
    for (int c = 0; c < NCOL; ++c) {
        const uint32_t key = v[c] ^ ((uint32_t)((int32_t)v[c] >> 31) & lc.fm[c]);
        ok &= (key - lc.lo[c]) <= lc.span[c];
    }
    return ok;
}

// One point at pixel (px, py) of tile t: the pixel slot of a mixed block, else
// the block total (an empty block keeps nothing: no polygon reads it).
template <bool AGG>
__device__ __forceinline__ void tl_splat(const TierLeanArgs& a, const LeanCols& lc, int t, int px, int py, float v) {
    const size_t b = (size_t)t * a.tr.bw * a.tr.bh + (size_t)(py >> 4) * a.tr.bw + (px >> 4);
    const uint32_t code = __ldg(a.tr.code + b);
    const bool fin = AGG && isfinite(v);
    const unsigned long long q = fin ? (unsigned long long)fixed_value(v, lc.scale) : 0ull;
    if ((code & kTierMixed) && code < kTierMulti) {
        const size_t at = (size_t)(code & ~kTierMixed) * 256 + (size_t)(py & 15) * 16 + (px & 15);
        atomicAdd(a.tr.pcnt + at, 1u);
        if (fin) atomicAdd(reinterpret_cast<unsigned long long*>(a.tr.psum + at), q);
    } else if (code != kTierEmpty) {
        atomicAdd(a.tr.bcnt + b, 1u);
        if (fin) atomicAdd(reinterpret_cast<unsigned long long*>(a.tr.bsum + b), q);
    }
}

template <int BLOCK, int NV, int NCOL, bool AGG>
__global__ void __launch_bounds__(BLOCK) k_tier_splat(TierLeanArgs a, LeanCols lc) {
    __shared__ float tx[kLeanMaxSplit], ty[kLeanMaxSplit];
    tl_stage_tiles<BLOCK>(a.ax, a.ay, tx, ty);
    __syncthreads();
    auto visit = [&](float x, float y, float val) {
        int cx, cy, px, py;
        if (tl_inner(x, a.ax, tx, cx, px) & tl_inner(y, a.ay, ty, cy, py))
            tl_splat<AGG>(a, lc, cy * a.ax.split + cx, px, py, val);
        else
            tl_hits(a.ax, a.ay, tx, ty, x, y, [&](int hx, int hy, int qx, int qy) {
                tl_splat<AGG>(a, lc, hy * a.ax.split + hx, qx, qy, val);
            });
    };
    const uint2* aggr2 = lc.aggr_col;
    const uint64_t npairs = a.n >> 1;
    constexpr uint64_t kPerIter = (uint64_t)BLOCK * NV;
    const uint64_t warp_ofs = (uint64_t)(threadIdx.x >> 5) * 32 * NV;
    const uint64_t lane_ofs = warp_ofs + (threadIdx.x & 31);
    for (uint64_t base = (uint64_t)blockIdx.x * kPerIter; base < npairs; base += (uint64_t)gridDim.x * kPerIter) {
        if (!tl_zone<NV>(a, base + warp_ofs)) continue;
        float4 p[NV];
        uint2 cv[NCOL > 0 ? NCOL : 1][NV];
        uint2 av[NV];
        #pragma unroll
        for (int k = 0; k < NV; ++k) {
            const uint64_t i = base + lane_ofs + (uint64_t)k * 32;
            const bool live = i < npairs;
            p[k] = live ? __ldcs(a.xy + i) : make_float4(NAN, NAN, NAN, NAN);
            #pragma unroll
            for (int c = 0; c < NCOL; ++c) cv[c][k] = live ? __ldcs(lc.col[c] + i) : make_uint2(0u, 0u);
            if (AGG) av[k] = (live && lc.aggr_ci < 0) ? __ldcs(aggr2 + i) : make_uint2(0u, 0u);
        }
        #pragma unroll
        for (int j = 0; j < 2 * NV; ++j) {
            const int k = j >> 1;
            const bool hi = (j & 1) != 0;
            uint32_t v[NCOL > 0 ? NCOL : 1];
            #pragma unroll
            for (int c = 0; c < NCOL; ++c) v[c] = hi ? cv[c][k].y : cv[c][k].x;
            if (!tl_pass<NCOL>(lc, v)) continue;
            float val = 0.f;
            if (AGG) {
                uint32_t raw = hi ? av[k].y : av[k].x;
                #pragma unroll
                for (int cc = 0; cc < NCOL; ++cc)
                    if (cc == lc.aggr_ci) raw = v[cc];
                val = agg_value(lc.aggr_typ, raw);
            }
            visit(hi ? p[k].z : p[k].x, hi ? p[k].w : p[k].y, val);
        }
    }
    // the last point of an odd-sized table
    if ((a.n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const uint64_t i = a.n - 1;
        const float2 q = __ldg(reinterpret_cast<const float2*>(a.xy) + i);
        uint32_t v[NCOL > 0 ? NCOL : 1];
        #pragma unroll
        for (int c = 0; c < NCOL; ++c) v[c] = __ldg(reinterpret_cast<const uint32_t*>(lc.col[c]) + i);
        if (tl_pass<NCOL>(lc, v)) {
            float fv = 0.f;
            if (AGG) {
                uint32_t raw = lc.aggr_ci < 0 ? __ldg(reinterpret_cast<const uint32_t*>(aggr2) + i) : 0u;
                #pragma unroll
                for (int cc = 0; cc < NCOL; ++cc)
                    if (cc == lc.aggr_ci) raw = v[cc];
                fv = agg_value(lc.aggr_typ, raw);
            }
            visit(q.x, q.y, fv);
        }
    }
}

using TierLeanKernel = void (*)(TierLeanArgs, LeanCols);

struct TlShape {
    int block;
    int nv;
};
constexpr TlShape kTlShapes[] = {{512, 2}, {256, 4}, {1024, 2}};
constexpr int kNumTlShapes = (int)(sizeof(kTlShapes) / sizeof(kTlShapes[0]));

template <int NCOL, bool AGG>
TierLeanKernel pick_tl(int shape) {
    switch (shape) {
        case 0: return k_tier_splat<512, 2, NCOL, AGG>;
        case 1: return k_tier_splat<256, 4, NCOL, AGG>;
        default: return k_tier_splat<1024, 2, NCOL, AGG>;
    }
}

template <bool AGG>
TierLeanKernel pick_tl_ncol(int ncol, int shape) {
    switch (ncol) {
        case 0: return pick_tl<0, AGG>(shape);
        case 1: return pick_tl<1, AGG>(shape);
        case 2: return pick_tl<2, AGG>(shape);
        case 3: return pick_tl<3, AGG>(shape);
        case 4: return pick_tl<4, AGG>(shape);
        default: return nullptr;
    }
}

}  // namespace

int tier_lean_shapes() { return kNumTlShapes; }

bool launch_tier_lean(int shape, const TierLeanArgs& a, const LeanCols& lc, int sms, cudaStream_t st) {
    if (shape < 0 || shape >= kNumTlShapes || lc.ncol < 0 || lc.ncol > 4) return false;
    if (a.ax.split > kLeanMaxSplit || a.ay.split > kLeanMaxSplit) return false;
    const bool agg = lc.aggr != 0;
    if (agg && (!a.tr.bsum || !a.tr.psum)) return false;
    TierLeanKernel k = agg ? pick_tl_ncol<true>(lc.ncol, shape) : pick_tl_ncol<false>(lc.ncol, shape);
    if (!k) return false;
    const int block = kTlShapes[shape].block;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, block, 0) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    const uint64_t per_iter = (uint64_t)block * kTlShapes[shape].nv;
    const uint64_t need = ((a.n >> 1) + per_iter - 1) / per_iter;
    const uint64_t blocks = std::min<uint64_t>((uint64_t)sms * per_sm, std::max<uint64_t>(need, 1));
    k<<<(unsigned)blocks, block, 0, st>>>(a, lc);
    ++g_kernel_launches;
    return true;
}

}  // namespace rj
