// rj_splat_bins.cu -- point counts onto a large one-tile canvas through bins
// instead of one atomic per point in L2 (which takes about 170 G points/s,
// whatever the loads do).
//
// The canvas is cut into bins of 128 x 128 pixels, whose counts fit shared
// memory three times per SM.  k_bin_points orders 16,384 points by bin in
// shared memory (count, scan, place) and writes their 14-bit pixel offsets out
// in one linear copy, with the starts of its bins; a bin's run begins on a
// multiple of four points (one 8-byte load later).  k_bin_counts takes one bin,
// counts its runs of all chunks in shared memory, with as many lanes to a run
// as the bin's runs are long, and adds them to the canvas with plain stores;
// bins that hold far more than their share are split over several blocks, which
// then add atomically (k_bin_plan).  So a point costs 8 bytes read, two written
// and two read again, and its atomics stay on the SM.
//
// Measured (4000 x 4000 pixels, 1,024 bins, points 80 % in eight clusters): point
// pass 2.64 ms for 500M points against 3.05 with atomics in L2, 531 us against
// 587 for 100M, 213 against 187 for 30M.  Of 491 us for 100M k_bin_points is
// 299, bound by shared-memory wavefronts (16 per 32 points: two atomics with
// conflicts, the placing, the detour through s_what), and k_bin_counts 192, bound
// by the latency of its short runs; with a full warp per run, whatever its
// length, it took 341.
//
// The predicates and the exact snapped pixel are those of rj_splat_kernels.cu.
#include <atomic>

#include "rj_label_core.cuh"

namespace rj {

namespace {

constexpr int kBinBits = 7;                         // log2 of a bin's side
constexpr int kBinSide = 1 << kBinBits, kBinPix = kBinSide * kBinSide;
constexpr int kMaxBins = 1536;
constexpr int kChunk = 16384;                       // points ordered at a time
constexpr int kOut = kChunk + 3 * kMaxBins;         // ... with the runs padded to fours
constexpr int kBT = 512;                            // threads, both passes
constexpr int kPairs = kChunk / 2 / kBT;            // pairs per thread
constexpr uint32_t kNoPixel = 0xFFFFu;              // padding
constexpr int kCountBlocks = 3;                     // blocks per SM of k_bin_counts

struct BinArgs {
    int nbx, nb, nchunks;
    int out;                        // points a chunk's padded runs may take
    uint16_t* data;                 // [nchunks][out] pixel offsets, by bin
    uint16_t* starts;               // [nb + 1][nchunks] where a bin's run starts, in fours
    unsigned* total;                // [nb] points of a bin
    unsigned* ctr;                  // [2] items handed out, items
    uint32_t* items;                // bin << 12 | part of it
    uint32_t* parts;                // [nb] parts of a bin
};

template <int NCOL>
__global__ void __launch_bounds__(kBT, 2) k_bin_points(SplatLeanArgs a, LeanCols lc, BinArgs b) {
    extern __shared__ __align__(16) char s_raw[];
    uint2* s_what = reinterpret_cast<uint2*>(s_raw);                        // [kChunk / 2] bin << 14 | pixel
    uint16_t* s_out = reinterpret_cast<uint16_t*>(s_raw + kChunk * 4);      // [kOut]
    uint32_t* s_count = reinterpret_cast<uint32_t*>(s_raw + kChunk * 4 + kOut * 2);   // [kMaxBins]
    __shared__ uint32_t s_warp[kBT / 32];
    constexpr int kMine = kMaxBins / kBT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float Hx = __fmul_rn(a.col0.z, (float)kSub), Hy = __fmul_rn(a.row0.z, (float)kSub);
    const uint64_t npairs = a.n >> 1;
    uint32_t mine[kMine] = {};
    for (int chunk = blockIdx.x; chunk < b.nchunks; chunk += gridDim.x) {
        for (int i = threadIdx.x; i < kMaxBins; i += kBT) s_count[i] = 0u;
        for (int i = threadIdx.x; i < b.out / 8; i += kBT)
            reinterpret_cast<uint4*>(s_out)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        __syncthreads();
        for (int h = 0; h < kPairs; h += 4) {
            const int local = (warp * kPairs + h) * 32 + lane;
            const uint64_t first = (uint64_t)chunk * (kChunk / 2) + (uint64_t)(local - lane);
            const bool meets = tl_zone<4>(a, first);
            float4 p[4];
            uint2 cv[NCOL > 0 ? NCOL : 1][4];
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t i = first + (uint64_t)k * 32 + lane;
                const bool live = meets && i < npairs;
                p[k] = live ? __ldcs(a.xy + i) : make_float4(NAN, NAN, NAN, NAN);
                #pragma unroll
                for (int c = 0; c < NCOL; ++c) cv[c][k] = live ? __ldcs(lc.col[c] + i) : make_uint2(0u, 0u);
            }
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t w[2];
                #pragma unroll
                for (int j = 0; j < 2; ++j) {
                    bool ok = true;
                    #pragma unroll
                    for (int c = 0; c < NCOL; ++c) {
                        const uint32_t v = j ? cv[c][k].y : cv[c][k].x;
                        const uint32_t key = v ^ ((uint32_t)((int32_t)v >> 31) & lc.fm[c]);
                        ok &= (key - lc.lo[c]) <= lc.span[c];
                    }
                    const int px = snapped_pixel(j ? p[k].z : p[k].x, a.col0.x, a.col0.y, Hx);
                    const int py = snapped_pixel(j ? p[k].w : p[k].y, a.row0.x, a.row0.y, Hy);
                    ok = ok && (unsigned)px < (unsigned)a.resx && (unsigned)py < (unsigned)a.resy;
                    const uint32_t bin = (uint32_t)((py >> kBinBits) * b.nbx + (px >> kBinBits));
                    const uint32_t at = (uint32_t)((py & (kBinSide - 1)) << kBinBits | (px & (kBinSide - 1)));
                    w[j] = ok ? bin << (2 * kBinBits) | at : 0xFFFFFFFFu;
                    if (ok) atomicAdd(s_count + bin, 1u);
                }
                s_what[local + 32 * k] = make_uint2(w[0], w[1]);
            }
        }
        __syncthreads();
        // counts -> starts (kMine neighbouring bins a thread)
        uint32_t v[kMine], sum = 0u;
        #pragma unroll
        for (int u = 0; u < kMine; ++u) {
            v[u] = s_count[threadIdx.x * kMine + u];
            mine[u] += v[u];
            v[u] = (v[u] + 3u) & ~3u;
            sum += v[u];
        }
        uint32_t incl = sum;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t at = incl - sum, total = 0u;
        #pragma unroll
        for (int w = 0; w < kBT / 32; ++w) {
            at += w < warp ? s_warp[w] : 0u;
            total += s_warp[w];
        }
        #pragma unroll
        for (int u = 0; u < kMine; ++u) {
            const int bin = (int)threadIdx.x * kMine + u;
            s_count[bin] = at;
            if (bin < b.nb) b.starts[(size_t)bin * b.nchunks + chunk] = (uint16_t)(at >> 2);
            at += v[u];
        }
        if (threadIdx.x == 0) b.starts[(size_t)b.nb * b.nchunks + chunk] = (uint16_t)(total >> 2);
        __syncthreads();
        #pragma unroll 8
        for (int h = 0; h < kPairs; ++h) {
            const uint2 w = s_what[(warp * kPairs + h) * 32 + lane];
            if (w.x != 0xFFFFFFFFu) s_out[atomicAdd(s_count + (w.x >> (2 * kBinBits)), 1u)] = (uint16_t)(w.x & (kBinPix - 1));
            if (w.y != 0xFFFFFFFFu) s_out[atomicAdd(s_count + (w.y >> (2 * kBinBits)), 1u)] = (uint16_t)(w.y & (kBinPix - 1));
        }
        __syncthreads();
        uint4* out = reinterpret_cast<uint4*>(b.data + (size_t)chunk * b.out);
        for (uint32_t i = threadIdx.x; i * 8 < total; i += kBT) out[i] = reinterpret_cast<const uint4*>(s_out)[i];
        __syncthreads();
    }
    #pragma unroll
    for (int u = 0; u < kMine; ++u)
        if (mine[u]) atomicAdd(b.total + threadIdx.x * kMine + u, mine[u]);
}

// One block: the work items.  A bin with up to an even share of the points per
// resident block is one item; a heavier one is cut into parts of that size, a
// part being a range of the chunks.
__global__ void __launch_bounds__(1024) k_bin_plan(BinArgs b, int resident) {
    __shared__ unsigned s_sum;
    if (threadIdx.x == 0) s_sum = 0u;
    __syncthreads();
    constexpr int kMine = (kMaxBins + 1023) / 1024;
    unsigned t[kMine], sum = 0u;
    #pragma unroll
    for (int u = 0; u < kMine; ++u) {
        const int bin = (int)threadIdx.x + u * 1024;
        t[u] = bin < b.nb ? b.total[bin] : 0u;
        sum += t[u];
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, sum);
    __syncthreads();
    const unsigned share = max(s_sum / (unsigned)resident + 1u, 4u * kBinPix);
    #pragma unroll
    for (int u = 0; u < kMine; ++u) {
        const int bin = (int)threadIdx.x + u * 1024;
        if (t[u] == 0u) continue;
        const unsigned parts = min(t[u] / share + 1u, (unsigned)b.nchunks);
        b.parts[bin] = parts;
        const unsigned first = atomicAdd(b.ctr + 1, parts);
        for (unsigned q = 0; q < parts; ++q) b.items[first + q] = (uint32_t)bin << 12 | q;
    }
}

__global__ void __launch_bounds__(kBT, kCountBlocks) k_bin_counts(SplatLeanArgs a, BinArgs b) {
    extern __shared__ __align__(16) uint32_t s_can[];   // [kBinPix]
    __shared__ unsigned s_item;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned nitems = b.ctr[1];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(b.ctr, 1u);
        for (int i = threadIdx.x; i < kBinPix / 4; i += kBT) reinterpret_cast<uint4*>(s_can)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        if (s_item >= nitems) return;
        const uint32_t item = b.items[s_item];
        const int bin = (int)(item >> 12), part = (int)(item & 4095u), parts = (int)b.parts[bin];
        const int c0 = (int)((long long)b.nchunks * part / parts), c1 = (int)((long long)b.nchunks * (part + 1) / parts);
        const uint16_t* from = b.starts + (size_t)bin * b.nchunks;
        const uint16_t* to = from + b.nchunks;
        // lanes to a run: half the fours of an average run, so that a run takes
        // two or three turns and few lanes idle
        const unsigned mean = b.total[bin] / (unsigned)b.nchunks >> 3;
        const int lg = mean ? min(31 - __clz(mean), 5) : 0, L = 1 << lg;
        // chunks a warp takes at a time (few chunks are spread over all warps)
        const int g = min(max((c1 - c0 + kBT / 32 - 1) / (kBT / 32), 1), 32);
        const int stride = kBT / 32 * g;
        const auto bounds = [&](int cc, int& s, int& e) {
            const bool has = lane < g && cc + lane < c1;
            s = has ? (int)__ldg(from + cc + lane) : 0;
            e = has ? (int)__ldg(to + cc + lane) : 0;
        };
        const auto add = [&](uint32_t w) {
            if ((w & 0xFFFFu) != kNoPixel) atomicAdd(s_can + (w & 0xFFFFu), 1u);
            if (w >> 16 != kNoPixel) atomicAdd(s_can + (w >> 16), 1u);
        };
        const uint2 none = make_uint2(~0u, ~0u);
        int c = c0 + warp * g, s, e;
        bounds(c, s, e);
        while (c < c1) {
            int s2, e2;
            bounds(c + stride, s2, e2);
            for (int k = 0; k < g; k += 32 >> lg) {
                const int run = (k + (lane >> lg)) & 31;
                const uint2* d = reinterpret_cast<const uint2*>(b.data + (size_t)(c + run) * b.out);
                const int first = __shfl_sync(0xffffffffu, s, run), last = __shfl_sync(0xffffffffu, e, run);
                for (int i = first + (lane & (L - 1)); __any_sync(0xffffffffu, i < last); i += 2 * L) {
                    const uint2 w0 = i < last ? __ldcs(d + i) : none, w1 = i + L < last ? __ldcs(d + i + L) : none;
                    add(w0.x);
                    add(w0.y);
                    add(w1.x);
                    add(w1.y);
                }
            }
            c += stride;
            s = s2;
            e = e2;
        }
        __syncthreads();
        uint32_t* can = a.canvas_c + ((size_t)(bin / b.nbx) * a.resx + bin % b.nbx) * kBinSide;
        #pragma unroll 8
        for (int i = threadIdx.x; i < kBinPix; i += kBT) {
            const uint32_t n = s_can[i];
            uint32_t* at = can + (size_t)(i >> kBinBits) * a.resx + (i & (kBinSide - 1));
            if (n && parts == 1) *at += n;
            else if (n) atomicAdd(at, n);
        }
        __syncthreads();
    }
}

// the last point of an odd-sized table, straight into the canvas
__global__ void k_bin_last(SplatLeanArgs a, LeanCols lc) {
    const uint64_t i = a.n - 1;
    const float2 q = __ldg(reinterpret_cast<const float2*>(a.xy) + i);
    for (int c = 0; c < lc.ncol; ++c) {
        const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(lc.col[c]) + i);
        const uint32_t key = v ^ ((uint32_t)((int32_t)v >> 31) & lc.fm[c]);
        if ((key - lc.lo[c]) > lc.span[c]) return;
    }
    const int px = snapped_pixel(q.x, a.col0.x, a.col0.y, __fmul_rn(a.col0.z, (float)kSub));
    const int py = snapped_pixel(q.y, a.row0.x, a.row0.y, __fmul_rn(a.row0.z, (float)kSub));
    if ((unsigned)px < (unsigned)a.resx && (unsigned)py < (unsigned)a.resy)
        atomicAdd(a.canvas_c + (size_t)py * a.resx + px, 1u);
}

// points per round: bounds the scratch (two bytes a point)
constexpr uint64_t kRound = 1ull << 27;
constexpr size_t kPointSmem = (size_t)kChunk * 4 + kOut * 2 + kMaxBins * 4;
constexpr size_t kCountSmem = (size_t)kBinPix * 4;
constexpr int kMaxParts = 4096;        // parts of a bin (12 bits of an item)

int bins_x(int resx) { return (resx + kBinSide - 1) >> kBinBits; }
long long bins_of(int resx, int resy) { return (long long)bins_x(resx) * bins_x(resy); }
int out_of(int nb) { return kChunk + 3 * ((nb + 7) & ~7); }
size_t up16(size_t v) { return (v + 15) & ~(size_t)15; }

using BinKernel = void (*)(SplatLeanArgs, LeanCols, BinArgs);
BinKernel bin_kernel(int ncol) {
    switch (ncol) {
        case 0: return k_bin_points<0>;
        case 1: return k_bin_points<1>;
        case 2: return k_bin_points<2>;
        case 3: return k_bin_points<3>;
        default: return k_bin_points<4>;
    }
}

}  // namespace

bool splat_bins_fit(int resx, int resy, int sms, bool agg) {
    return !agg && bins_of(resx, resy) <= kMaxBins && sms * kCountBlocks < kMaxParts;
}

size_t splat_bins_bytes(int resx, int resy, int sms, uint64_t n) {
    const size_t chunks = (size_t)((std::min(n, kRound) + kChunk - 1) / kChunk), nb = (size_t)bins_of(resx, resy);
    return chunks * out_of((int)nb) * 2 + up16(chunks * (nb + 1) * 2) + up16((nb + 2) * 4) + up16(nb * 4) +
           (nb + (size_t)sms * kCountBlocks) * 4;
}

// `scratch` holds splat_bins_bytes (16-byte aligned)
bool launch_splat_bins(const SplatLeanArgs& a_in, const LeanCols& lc_in, void* scratch, int sms, cudaStream_t st) {
    if (lc_in.ncol < 0 || lc_in.ncol > 4) return false;
    const BinKernel points = bin_kernel(lc_in.ncol);
    if (allow_smem(reinterpret_cast<const void*>(points), kPointSmem) != cudaSuccess ||
        allow_smem(reinterpret_cast<const void*>(k_bin_counts), kCountSmem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    for (uint64_t r0 = 0; r0 < a_in.n; r0 += kRound) {
        SplatLeanArgs a = a_in;
        LeanCols lc = lc_in;
        a.n = std::min(kRound, a_in.n - r0);
        a.xy += r0 / 2;
        a.zrow0 += r0;
        for (int c = 0; c < lc.ncol; ++c) lc.col[c] += r0 / 2;
        BinArgs b{};
        b.nbx = bins_x(a.resx);
        b.nb = (int)bins_of(a.resx, a.resy);
        b.out = out_of(b.nb);
        b.nchunks = (int)(((a.n & ~1ull) + kChunk - 1) / kChunk);
        if (b.nchunks) {
            char* p = (char*)scratch;
            b.data = (uint16_t*)p;
            p += (size_t)b.nchunks * b.out * 2;
            b.starts = (uint16_t*)p;
            p += up16((size_t)b.nchunks * (b.nb + 1) * 2);
            b.ctr = (unsigned*)p;
            b.total = b.ctr + 2;
            p += up16(((size_t)b.nb + 2) * 4);
            b.parts = (uint32_t*)p;
            p += up16((size_t)b.nb * 4);
            b.items = (uint32_t*)p;
            if (cudaMemsetAsync(b.ctr, 0, ((size_t)b.nb + 2) * 4, st) != cudaSuccess) return false;
            points<<<std::min(b.nchunks, sms * 2), kBT, kPointSmem, st>>>(a, lc, b);
            k_bin_plan<<<1, 1024, 0, st>>>(b, sms * kCountBlocks);
            k_bin_counts<<<sms * kCountBlocks, kBT, kCountSmem, st>>>(a, b);
            g_kernel_launches += 3;
        }
        if (a.n & 1) {
            k_bin_last<<<1, 1, 0, st>>>(a, lc);
            ++g_kernel_launches;
        }
    }
    return true;
}

}  // namespace rj
