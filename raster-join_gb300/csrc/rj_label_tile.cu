// rj_label_tile.cu -- lean label pass of a one-tile canvas without filters: a
// count, or a sum, per polygon (the reference renders every point and then
// every polygon, RasterJoin.cpp:91-194, points.vert:138-159, polygon.frag:12-27).
//
// Every point takes the exact pixel (rj_lean.cuh), written with as few
// operations as that allows: adding 1.5 * 2^23 to the window coordinate * 256
// rounds it to the integer the snap asks for and leaves it in the low mantissa
// bits, so that no conversion (a quarter-rate instruction) and no clamp is
// needed, and one unsigned compare per axis rejects everything off the canvas,
// NaN and infinities included.  The code of the pixel's block of 2^bs x 2^bs
// pixels (the one polygon all its pixels hold, "none", or "mixed") comes from
// shared memory; only points of mixed blocks read the pixel's label from L2,
// all of a thread's points before the first is used.
//
// What bounds it is the L1 / shared-memory pipe (93 % of its rate with 32 x 32
// blocks): 32 random points take about three wavefronts for the code, three for
// the histogram add, two for their locations and one for every label read.
// 16 x 16 blocks on one block of 1024 threads per SM (125 KB of codes for a
// 4000 x 4000 canvas; 15 % of the points read a label) beat 32 x 32 blocks on
// two (28 %).  2B points, 260 Voronoi cells at 10 m, count: 2.88 ms = 5.56 TB/s;
// with conversions, a clamp and a flat label map 3.13 ms.  Loading the next
// points while the labels arrive made it slower (3.45 ms), as did queueing the
// points of mixed blocks (3.6 to 4.9 ms).
#include "rj_label_core.cuh"

namespace rj {

// Block codes of 2^bs x 2^bs pixels from the canvas's 16 x 16 codes, a thread
// per block.
__global__ void k_label_blocks(TierArgs tr, int bs, int nbx, int nby, int P, uint16_t* __restrict__ codes) {
    const int f = 1 << (bs - 4), n = nbx * nby;
    if (blockIdx.x == 0 && threadIdx.x == 0) codes[n] = kEmptyLabel;   // off the canvas
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const int y0 = s / nbx * f, x0 = (s - s / nbx * nbx) * f;
        const int x1 = min(x0 + f, tr.bw), y1 = min(y0 + f, tr.bh);
        const uint32_t first = __ldg(tr.code + y0 * tr.bw + x0);
        bool same = first < (uint32_t)P || first == kTierEmpty;
        for (int y = y0; y < y1; ++y)
            for (int x = x0; x < x1; ++x) same &= __ldg(tr.code + y * tr.bw + x) == first;
        codes[s] = same ? (uint16_t)first : kCodeMixed;   // kTierEmpty -> kEmptyLabel
    }
}

void launch_label_blocks(const TierArgs& tr, int bs, int nbx, int nby, int P, uint16_t* codes, int sms, cudaStream_t st) {
    const int blocks = std::max(1, std::min((nbx * nby + 255) / 256, sms * 8));
    k_label_blocks<<<blocks, 256, 0, st>>>(tr, bs, nbx, nby, P, codes);
    ++g_kernel_launches;
}

// pixel * 256 of a coordinate (>= the canvas size * 256 when it lies outside)
__device__ __forceinline__ uint32_t pixel256(float v, const TileAxis& x, float t) {
    const float w = __fadd_rn(__fmul_rn(x.H, __fadd_rn(__fmul_rn(x.s, v), t)), x.H);   // window coordinate * 256
    return __float_as_uint(__fadd_rn(w, 12582912.0f)) - kCellMagic;
}

// ONE: the blocks are the canvas's own (bs == 4) and a mixed block's labels
// lie at its own place.
template <int BLOCK, int NV, int MINB, bool AGG, bool ONE>
__global__ void __launch_bounds__(BLOCK, MINB) k_label_tile(LabelPointArgs a, LeanCols lc) {
    extern __shared__ uint32_t s_words[];
    constexpr int HW = AGG ? 3 : 1;
    uint32_t* s_hist = s_words + a.cell_words;                        // lc.copies x HW x P
    {
        const uint32_t* g = reinterpret_cast<const uint32_t*>(a.cells);
        for (int i = threadIdx.x; i < a.cell_words; i += BLOCK) s_words[i] = __ldg(g + i);
        for (int i = threadIdx.x; i < lc.copies * HW * a.P; i += BLOCK) s_hist[i] = 0u;
    }
    __syncthreads();
    const uint16_t* sc = reinterpret_cast<const uint16_t*>(s_words);
    const uint32_t P = (uint32_t)a.P;
    uint32_t* hist = s_hist + ((threadIdx.x >> 5) & (lc.copies - 1)) * HW * a.P;
    const float tx = __ldg(a.ax.xf).y, ty = __ldg(a.ay.xf).y;
    const uint32_t wx = (uint32_t)a.ax.res << 8, wy = (uint32_t)a.ay.res << 8;
    const int sh = 8 + (ONE ? 4 : a.bs);
    const uint32_t nbx = (uint32_t)a.cnx, none = nbx * (uint32_t)a.cny;

    // offset of pixel (px, py), both * 256, in its 16 x 16 block
    auto offset = [](uint32_t px, uint32_t py) { return (py >> 4 & 0xF0u) | (px >> 8 & 15u); };
    // entry of the code map: past its end ("none") off the canvas
    auto block_of = [&](uint32_t px, uint32_t py) {
        const uint32_t s = (py >> sh) * nbx + (px >> sh);
        return px < wx && py < wy ? s : none;
    };
    const uint64_t npairs = a.n >> 1;
    constexpr uint64_t kPerIter = (uint64_t)BLOCK * NV;
    const uint64_t warp_ofs = (uint64_t)(threadIdx.x >> 5) * 32 * NV;
    auto iterate = [&](uint64_t base, bool full) {
        float4 p[NV];
        uint2 av[NV];
        #pragma unroll
        for (int k = 0; k < NV; ++k) {
            const uint64_t i = base + warp_ofs + (threadIdx.x & 31) + (uint64_t)k * 32;
            const bool live = full || i < npairs;
            p[k] = live ? __ldcs(a.xy + i) : make_float4(NAN, NAN, NAN, NAN);
            if (AGG) av[k] = live ? __ldcs(lc.aggr_col + i) : make_uint2(0u, 0u);
        }
        uint32_t lab[2 * NV], ofs[2 * NV];
        #pragma unroll
        for (int j = 0; j < 2 * NV; ++j) {
            const uint32_t px = pixel256((j & 1) ? p[j >> 1].z : p[j >> 1].x, a.ax, tx);
            const uint32_t py = pixel256((j & 1) ? p[j >> 1].w : p[j >> 1].y, a.ay, ty);
            const uint32_t s = block_of(px, py);
            lab[j] = sc[s];
            ofs[j] = offset(px, py);
            if (ONE) {
                const uint16_t* at = a.tr.plabel + (s << 8 | ofs[j]);
                if (lab[j] == kCodeMixed) lab[j] = __ldg(at);
            } else {
                const uint32_t* at = a.tr.code + (py >> 12) * (uint32_t)a.tr.bw + (px >> 12);
                if (lab[j] == kCodeMixed) lab[j] = __ldg(at);
            }
        }
        if (!ONE) {
            #pragma unroll
            for (int j = 0; j < 2 * NV; ++j) {
                const uint16_t* at = a.tr.plabel + ((size_t)(lab[j] & ~kTierMixed) << 8 | ofs[j]);
                if (lab[j] >= kTierMixed && lab[j] < kTierMulti) lab[j] = __ldg(at);
            }
        }
        #pragma unroll
        for (int j = 0; j < 2 * NV; ++j)
            if (lab[j] < P)
                label_add<AGG>(hist, P, lc, lab[j],
                               AGG ? agg_value(lc.aggr_typ, (j & 1) ? av[j >> 1].y : av[j >> 1].x) : 0.f);
    };
    for (uint64_t base = (uint64_t)blockIdx.x * kPerIter; base < npairs; base += (uint64_t)gridDim.x * kPerIter) {
        if (!tl_zone<NV>(a, base + warp_ofs)) continue;
        if (base + kPerIter <= npairs) iterate(base, true);
        else iterate(base, false);
    }
    // the last point of an odd-sized table
    if ((a.n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const float2 q = __ldg(reinterpret_cast<const float2*>(a.xy) + (a.n - 1));
        const uint32_t px = pixel256(q.x, a.ax, tx), py = pixel256(q.y, a.ay, ty);
        const uint32_t s = block_of(px, py);
        uint32_t c = sc[s];
        if (c == kCodeMixed) {
            uint32_t slot = s;
            c = kTierMixed;
            if (!ONE) c = __ldg(a.tr.code + (py >> 12) * (uint32_t)a.tr.bw + (px >> 12)), slot = c & ~kTierMixed;
            if (c >= kTierMixed && c < kTierMulti) c = __ldg(a.tr.plabel + ((size_t)slot << 8 | offset(px, py)));
        }
        if (c < P)
            label_add<AGG>(hist, P, lc, c,
                           AGG ? agg_value(lc.aggr_typ, __ldg(reinterpret_cast<const uint32_t*>(lc.aggr_col) + (a.n - 1))) : 0.f);
    }
    __syncthreads();
    label_flush<BLOCK, AGG>(a, lc, s_hist);
}

namespace {

struct TileShape {
    int block, nv;
};
constexpr TileShape kTileShapes[] = {{1024, 4}, {1024, 4}, {512, 4}, {1024, 2}};
constexpr int kNumTileShapes = (int)(sizeof(kTileShapes) / sizeof(kTileShapes[0]));

template <bool AGG, bool ONE>
LabelKernel tile_kernel(int shape) {
    switch (shape) {
        case 0: return k_label_tile<1024, 4, 1, AGG, ONE>;
        case 1: return k_label_tile<1024, 4, 2, AGG, ONE>;   // two blocks per SM: 32 registers
        case 2: return k_label_tile<512, 4, 3, AGG, ONE>;
        case 3: return k_label_tile<1024, 2, 2, AGG, ONE>;
        default: return nullptr;
    }
}

// histogram copies: a power of two up to the warps of the block, within 36 KB
int tile_copies(int shape, int P, bool agg) {
    const size_t per = (size_t)P * (agg ? 3 : 1) * 4;
    int copies = 1;
    while (copies * 2 <= kTileShapes[shape].block / 32 && per * copies * 2 <= 36 * 1024) copies *= 2;
    return copies;
}

}  // namespace

int label_tile_shapes() { return kNumTileShapes; }

size_t label_tile_smem(int shape, int cell_words, int P, bool agg) {
    return (size_t)cell_words * 4 + (size_t)tile_copies(shape, P, agg) * P * (agg ? 3 : 1) * 4;
}

bool launch_label_tile(int shape, const LabelPointArgs& a, const LeanCols& lc_in, int sms, cudaStream_t st) {
    if (shape < 0 || shape >= kNumTileShapes || lc_in.ncol != 0 || a.ax.split != 1 || a.ay.split != 1) return false;
    const bool agg = lc_in.aggr != 0, one = a.bs == 4 && a.tr.own_place;
    LabelKernel k = agg ? (one ? tile_kernel<true, true>(shape) : tile_kernel<true, false>(shape))
                        : (one ? tile_kernel<false, true>(shape) : tile_kernel<false, false>(shape));
    LeanCols lc = lc_in;
    lc.copies = tile_copies(shape, a.P, agg);
    return launch_label_kernel(k, kTileShapes[shape].block, kTileShapes[shape].nv,
                               label_tile_smem(shape, a.cell_words, a.P, agg), a, lc, sms, st);
}

}  // namespace rj
