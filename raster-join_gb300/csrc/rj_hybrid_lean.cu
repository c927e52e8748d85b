// rj_hybrid_lean.cu -- lean point pass of the hybrid join (hybrid.glsl:224-300,
// HybridJoin::glJoin HybridJoin.cpp:87-195) over the hybrid canvas's polygon
// label map, and of the index join (index.glsl:186-248) over the classified
// grid's cell labels, with interval-form filters on up to four columns and
// an optional summed aggregate.
//
// Per point: the predicates, the hybrid canvas pixel (rasterize,
// hybrid.glsl:187-200), then the pixel's label through the block-code map in
// shared memory (the label map in L2 only for blocks whose pixels differ).
// A labelled pixel is inside exactly one polygon and away from every
// outline: the point goes to that polygon's histogram (plain shared-memory
// atomics, count and two-word fixed-point sum).  A pixel marked border (within
// the fp32 error radius of an outline, isBorder hybrid.glsl:174-185) sends the
// point to the exact test through the classified grid.
//
// Warps work alone.  The points that pass the filters (without filters: those
// whose block does not decide) are packed into the warp's queue and looked up
// 32 at a time; a batch only issues its label load, the next batch's turn uses
// it, and border points go on into a second queue that is tested 32 at a time.
//
// Measured (100M points, filters on four columns and avg, 24 B each, 260 cells):
// hybrid 512 us and index 508, 4.7 TB/s; 672 and 690 with block-wide queues,
// whose barriers came every iteration, and a label read each point waited for.
// Without filters 580 us.  What bounds it is the issue rate together with the
// latency that 32 warps of 64 registers can hide; three blocks of 512 threads
// per SM spill and take 850 us.
#include "rj_label_core.cuh"
#include "rj_point_core.cuh"

namespace rj {

namespace {

// Hist-like adapter for exact_probe: adds to the warp's histogram copy.
template <bool AGG>
struct LeanHist {
    uint32_t* hist;
    uint32_t P;
    const LeanCols* lc;
    __device__ __forceinline__ void add(int p, float v) const { label_add<AGG>(hist, P, *lc, (uint32_t)p, v); }
};

// Where a point lies: 0 nowhere, 1 pixel (px, py), 2 the exact test decides.
//
// Hybrid canvas (mode 0): a labelled pixel lies in one polygon with no edge
// within the border radius (at least one pixel) of it, so every location
// within that slack of the pixel is inside the same polygon under the exact
// test.  The pixel therefore only has to be found to far better than a pixel,
// not bit for bit: one FMA per axis (error ~1e-4 px on a 4096-pixel canvas)
// instead of hybrid.glsl's two divisions.  Within 2 pixels of the canvas rim
// the exact rasterize decides, so the canvas bounds (half-open [-1, 1),
// hybrid.glsl:187-200) and NaN are handled exactly as before.
// Classified grid (mode 1): the cell of the exact test itself (index.glsl:
// 382-385, fp32 division, int() truncation).  A product with the reciprocal
// gives the same cell unless it comes within its error of an integer; there,
// and near the grid's rim, the division decides.
__device__ __forceinline__ int hyb_pixel(const HybLeanArgs& a, float x, float y, int& px, int& py) {
    if (a.mode == 0) {
        const float fx = fmaf(x, a.fast.x, a.fast.y), fy = fmaf(y, a.fast.z, a.fast.w);
        if (fx >= 2.0f && fx < (float)(a.h.resx - 2) && fy >= 2.0f && fy < (float)(a.h.resy - 2)) {
            px = (int)fx;
            py = (int)fy;
            return 1;
        }
        if (!hyb_rasterize(a.h, x, y, px, py)) return 0;
        return px >= a.h.resx || py >= a.h.resy ? 2 : 1;
    }
    const float dx = __fsub_rn(x, a.ix.lbx), dy = __fsub_rn(y, a.ix.lby);
    float gx = dx * a.fast.x, gy = dy * a.fast.z;
    const bool sure = fabsf(gx - floorf(gx) - 0.5f) < a.fast.y && fabsf(gy - floorf(gy) - 0.5f) < a.fast.y &&
                      gx >= 1.0f && gx < (float)(a.ix.res - 1) && gy >= 1.0f && gy < (float)(a.ix.res - 1);
    if (!sure) {
        gx = __fdiv_rn(dx, a.ix.csx);
        gy = __fdiv_rn(dy, a.ix.csy);
        if (!(gx > -1.0f && gx < (float)a.ix.res && gy > -1.0f && gy < (float)a.ix.res)) return 0;
    }
    px = (int)gx;
    py = (int)gy;
    return 1;
}

constexpr int kExactQueue = 64;         // border points of a warp: fewer than 32 left over plus a batch's

template <int NV>
__host__ __device__ constexpr int hyb_queue() { return 32 + 64 * NV; }   // left over + one iteration's points

}  // namespace

template <int BLOCK, int NV, int MINB, int NI, int NF, bool AGG>
__global__ void __launch_bounds__(BLOCK, MINB) k_hybrid_lean(HybLeanArgs a, LeanCols lc) {
    extern __shared__ uint32_t s_words[];
    constexpr int HW = AGG ? 3 : 1;
    constexpr int NCOL = NI + NF;
    constexpr int NA = NCOL > 0 ? NCOL : 1;
    constexpr int QC = hyb_queue<NV>();
    constexpr int W = BLOCK / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2* q = reinterpret_cast<float2*>(s_words) + warp * QC;
    float2* eq = reinterpret_cast<float2*>(s_words) + W * QC + warp * kExactQueue;
    uint32_t* s_vals = s_words + 2 * W * (QC + kExactQueue);
    uint32_t* qv = s_vals + warp * QC;                                  // AGG: their values (raw)
    uint32_t* ev = s_vals + W * QC + warp * kExactQueue;
    uint32_t* s_code = s_vals + (AGG ? W * (QC + kExactQueue) : 0);
    uint32_t* s_hist = s_code + a.code_words;                           // lc.copies x HW x P
    {
        const uint32_t* g = reinterpret_cast<const uint32_t*>(a.codes);
        for (int i = threadIdx.x; i < a.code_words; i += BLOCK) s_code[i] = __ldg(g + i);
        for (int i = threadIdx.x; i < lc.copies * HW * a.P; i += BLOCK) s_hist[i] = 0u;
    }
    __syncthreads();
    const uint16_t* sc = reinterpret_cast<const uint16_t*>(s_code);
    const uint32_t P = (uint32_t)a.P;
    const int resx = a.mode == 0 ? a.h.resx : a.ix.res;
    uint32_t* hist = s_hist + (warp & (lc.copies - 1)) * HW * a.P;
    const LeanHist<AGG> exact{hist, P, &lc};
    int qn = 0, en = 0;                 // queued points, queued border points (warp-uniform)
    bool tail = false, pending = false;
    // the batch in flight: its labels
    uint32_t lab = kEmptyLabel, raw1 = 0u;
    float2 at1 = make_float2(0.f, 0.f);

    // counts the batch in flight and sends off the last 32 (or fewer) queued points
    auto drain = [&]() {
        if (lab < P) label_add<AGG>(hist, P, lc, lab, AGG ? agg_value(lc.aggr_typ, raw1) : 0.f);
        const unsigned m = __ballot_sync(0xffffffffu, lab == kBorderLabel);
        if (lab == kBorderLabel) {
            const int s = en + __popc(m & ((1u << lane) - 1u));
            eq[s] = at1;
            if (AGG) ev[s] = raw1;
        }
        en += __popc(m);
        __syncwarp();
        while (en >= (tail ? 1 : 32)) {
            const int i = max(en - 32, 0) + lane;
            if (i < en) exact_probe(a.ix, eq[i].x, eq[i].y, AGG ? agg_value(lc.aggr_typ, ev[i]) : 0.f, exact);
            en = max(en - 32, 0);
            __syncwarp();
        }
        pending = qn > 0;
        lab = kEmptyLabel;
        const int first = max(qn - 32, 0);
        if (first + lane < qn) {
            at1 = q[first + lane];
            if (AGG) raw1 = qv[first + lane];
            int px, py;
            const int kind = hyb_pixel(a, at1.x, at1.y, px, py);
            if (kind == 1) {
                lab = NCOL > 0 ? sc[(py >> a.bs) * a.nbx + (px >> a.bs)] : kCodeMixed;
                if (lab == kCodeMixed) lab = __ldg(a.label + (size_t)py * resx + px);
            } else if (kind == 2) {
                lab = kBorderLabel;
            }
        }
        qn = first;
        __syncwarp();
    };

    const uint64_t npairs = a.n >> 1;
    constexpr uint64_t kPerIter = (uint64_t)BLOCK * NV;
    for (uint64_t base = (uint64_t)blockIdx.x * kPerIter + (uint64_t)warp * 32 * NV; !tail;
         base += (uint64_t)gridDim.x * kPerIter) {
        if (base >= npairs) {
            tail = true;
            // the last point of an odd-sized table
            if ((a.n & 1) && blockIdx.x == 0 && warp == 0) {
                const uint64_t i = a.n - 1;
                bool ok = true;
                if (lane == 0) {
                    uint32_t v[NA], raw = 0u;
                    #pragma unroll
                    for (int c = 0; c < NCOL; ++c) v[c] = __ldg(reinterpret_cast<const uint32_t*>(lc.col[c]) + i);
                    ok = cols_pass<NI, NF>(lc, v);
                    q[qn] = __ldg(reinterpret_cast<const float2*>(a.xy) + i);
                    if (AGG) {
                        if (lc.aggr_ci < 0) raw = __ldg(reinterpret_cast<const uint32_t*>(lc.aggr_col) + i);
                        #pragma unroll
                        for (int c = 0; c < NCOL; ++c)
                            if (c == lc.aggr_ci) raw = v[c];
                        qv[qn] = raw;
                    }
                }
                qn += __shfl_sync(0xffffffffu, ok ? 1 : 0, 0);
                __syncwarp();
            }
        } else if (tl_zone<NV>(a, base)) {
            float4 p[NV];
            uint2 cv[NA][NV];
            uint2 av[NV];
            #pragma unroll
            for (int k = 0; k < NV; ++k) {
                const uint64_t i = base + lane + (uint64_t)k * 32;
                const bool live = i < npairs;
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
            uint32_t push = 0u;   // points to queue
            #pragma unroll
            for (int j = 0; j < 2 * NV; ++j) {
                if (NCOL > 0) {
                    uint32_t v[NA];
                    #pragma unroll
                    for (int c = 0; c < NCOL; ++c) v[c] = (j & 1) ? cv[c][j >> 1].y : cv[c][j >> 1].x;
                    const bool ok = cols_pass<NI, NF>(lc, v) && base + lane + (uint64_t)(j >> 1) * 32 < npairs;
                    push |= ok ? 1u << j : 0u;
                } else {
                    int px, py;
                    const int kind = hyb_pixel(a, (j & 1) ? p[j >> 1].z : p[j >> 1].x, (j & 1) ? p[j >> 1].w : p[j >> 1].y,
                                               px, py);
                    uint32_t l = kind == 2 ? kBorderLabel : kEmptyLabel;
                    if (kind == 1) l = sc[(py >> a.bs) * a.nbx + (px >> a.bs)];
                    if (l < P) label_add<AGG>(hist, P, lc, l, AGG ? agg_value(lc.aggr_typ, value(j)) : 0.f);
                    push |= l == kCodeMixed || l == kBorderLabel ? 1u << j : 0u;
                }
            }
            // queue positions: one prefix sum over the lanes
            int incl = __popc(push);
            const int own = incl;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            int at = qn + incl - own;
            #pragma unroll
            for (int j = 0; j < 2 * NV; ++j)
                if ((push >> j) & 1u) {
                    q[at] = (j & 1) ? make_float2(p[j >> 1].z, p[j >> 1].w) : make_float2(p[j >> 1].x, p[j >> 1].y);
                    if (AGG) qv[at] = value(j);
                    ++at;
                }
            qn += __shfl_sync(0xffffffffu, incl, 31);
            __syncwarp();
        }
        while (qn >= 32 || (tail && (qn > 0 || pending))) drain();
    }
    __syncthreads();
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

// Block codes from a label map: one warp per block, eight pixels a load where
// rows and blocks allow (a 16 x 16 block is one load per lane).  On 4096 x 4096
// pixels 37 us with two-byte loads, 14 us now.
__global__ void k_block_codes(const uint16_t* __restrict__ label, int resx, int resy, int bs, int nbx, int nby,
                              uint16_t* __restrict__ codes) {
    const int lane = threadIdx.x & 31;
    const int B = 1 << bs;
    const int nb = nbx * nby;
    const bool wide = (resx & 7) == 0 && bs >= 3;
    for (int b = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); b < nb;
         b += (int)((gridDim.x * blockDim.x) >> 5)) {
        const int bx = b % nbx, by = b / nbx;
        const int x0 = bx << bs, y0 = by << bs;
        const int w = min(x0 + B, resx) - x0, h = min(y0 + B, resy) - y0;
        const uint16_t first = __ldg(label + (size_t)y0 * resx + x0);
        bool same = true;
        if (wide) {
            const uint32_t both = first * 0x10001u;
            const int w8 = w >> 3;
            for (int i = lane; i < w8 * h; i += 32) {
                const int yy = w == B ? i >> (bs - 3) : i / w8;
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(label + (size_t)(y0 + yy) * resx + x0) + (i - yy * w8));
                same &= v.x == both && v.y == both && v.z == both && v.w == both;
            }
        } else {
            for (int i = lane; i < w * h; i += 32) {
                const int yy = y0 + i / w, xx = x0 + i % w;
                same &= (__ldg(label + (size_t)yy * resx + xx) == first);
            }
        }
        same = __all_sync(0xffffffffu, same);
        if (lane == 0) codes[b] = same ? first : kCodeMixed;
    }
}

void launch_block_codes(const uint16_t* label, int resx, int resy, int bs, int nbx, int nby, uint16_t* codes,
                        int sms, cudaStream_t st) {
    const long long warps = (long long)nbx * nby;
    long long blocks = (warps * 32 + 255) / 256;
    blocks = std::max(1LL, std::min(blocks, (long long)sms * 16));
    k_block_codes<<<(unsigned)blocks, 256, 0, st>>>(label, resx, resy, bs, nbx, nby, codes);
    ++g_kernel_launches;
}

// 16-bit cell labels of the classified grid for the lean pass (mode 1).
__global__ void k_cell_labels(const uint32_t* __restrict__ code, int ncells, uint16_t* __restrict__ label) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x) {
        const uint32_t v = __ldg(code + c);
        label[c] = v < kCodeList ? (uint16_t)v : (v == kCodeEmpty ? kEmptyLabel : kBorderLabel);
    }
}

void launch_cell_labels(const uint32_t* code, int ncells, uint16_t* label, int sms, cudaStream_t st) {
    const int blocks = std::max(1, std::min((ncells + 255) / 256, sms * 8));
    k_cell_labels<<<blocks, 256, 0, st>>>(code, ncells, label);
    ++g_kernel_launches;
}

// ---------------------------------------------------------------------------
namespace {

using HybKernel = void (*)(HybLeanArgs, LeanCols);

struct HybShape {
    int block, nv, minb;
};
constexpr HybShape kHybShapes[] = {{512, 2, 2}, {1024, 2, 1}};
constexpr int kNumHybShapes = (int)(sizeof(kHybShapes) / sizeof(kHybShapes[0]));

template <int NI, int NF, bool AGG>
HybKernel hyb_kernel(int shape) {
    switch (shape) {
        case 0: return k_hybrid_lean<512, 2, 2, NI, NF, AGG>;
        case 1: return k_hybrid_lean<1024, 2, 1, NI, NF, AGG>;
        default: return nullptr;
    }
}

template <bool AGG>
HybKernel hyb_kernel_cols(int shape, int ni, int nf) {
    switch (ni * 5 + nf) {
        case 0: return hyb_kernel<0, 0, AGG>(shape);
        case 1: return hyb_kernel<0, 1, AGG>(shape);
        case 2: return hyb_kernel<0, 2, AGG>(shape);
        case 3: return hyb_kernel<0, 3, AGG>(shape);
        case 4: return hyb_kernel<0, 4, AGG>(shape);
        case 5: return hyb_kernel<1, 0, AGG>(shape);
        case 6: return hyb_kernel<1, 1, AGG>(shape);
        case 7: return hyb_kernel<1, 2, AGG>(shape);
        case 8: return hyb_kernel<1, 3, AGG>(shape);
        case 10: return hyb_kernel<2, 0, AGG>(shape);
        case 11: return hyb_kernel<2, 1, AGG>(shape);
        case 12: return hyb_kernel<2, 2, AGG>(shape);
        case 15: return hyb_kernel<3, 0, AGG>(shape);
        case 16: return hyb_kernel<3, 1, AGG>(shape);
        case 20: return hyb_kernel<4, 0, AGG>(shape);
        default: return nullptr;
    }
}

int g_hyb_optin = -1;

// histogram copies: a power of two up to the warps of the block, within 32 KB
int hyb_copies(int shape, int P, bool agg) {
    const int warps = kHybShapes[shape].block / 32;
    int copies = 1;
    const size_t per = (size_t)P * (agg ? 3 : 1) * 4;
    while (copies * 2 <= warps && per * copies * 2 <= 32 * 1024) copies *= 2;
    return copies;
}

}  // namespace

int hybrid_lean_shapes() { return kNumHybShapes; }

size_t hybrid_lean_smem(int shape, int code_words, int P, bool agg) {
    if (shape < 0 || shape >= kNumHybShapes) return 0;
    const HybShape& s = kHybShapes[shape];
    const size_t queues = (size_t)(s.block / 32) * (32 + 64 * s.nv + kExactQueue) * (agg ? 12 : 8);
    return queues + (size_t)code_words * 4 + (size_t)hyb_copies(shape, P, agg) * P * (agg ? 3 : 1) * 4;
}

bool launch_hybrid_lean(int shape, const HybLeanArgs& a, const LeanCols& lc_in, int sms, cudaStream_t st) {
    if (shape < 0 || shape >= kNumHybShapes || lc_in.ncol < 0 || lc_in.ncol > 4) return false;
    const bool agg = lc_in.aggr != 0;
    const int ni = lc_in.nint, nf = lc_in.ncol - lc_in.nint;
    HybKernel k = agg ? hyb_kernel_cols<true>(shape, ni, nf) : hyb_kernel_cols<false>(shape, ni, nf);
    if (!k) return false;
    if (g_hyb_optin < 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_hyb_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    }
    LeanCols lc = lc_in;
    lc.copies = hyb_copies(shape, a.P, agg);
    const size_t smem = hybrid_lean_smem(shape, a.code_words, a.P, agg);
    if (smem > (size_t)g_hyb_optin) return false;
    if (allow_smem(reinterpret_cast<const void*>(k), smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int block = kHybShapes[shape].block;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, block, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    const uint64_t per_iter = (uint64_t)block * kHybShapes[shape].nv;
    const uint64_t need = ((a.n >> 1) + per_iter - 1) / per_iter;
    uint64_t blocks = std::min<uint64_t>((uint64_t)sms * per_sm, std::max<uint64_t>(need, 1));
    while (blocks < (uint64_t)sms * per_sm && a.n / blocks >= (1ull << 31)) ++blocks;
    if (a.n / blocks >= (1ull << 31)) return false;
    k<<<(unsigned)blocks, block, smem, st>>>(a, lc);
    ++g_kernel_launches;
    return true;
}

}  // namespace rj
