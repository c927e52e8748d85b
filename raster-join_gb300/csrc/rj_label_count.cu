// rj_label_count.cu -- the label pass that only counts (rj_label_core.cuh),
// the launcher of both forms, and the kernel that builds the cell codes.
#include "rj_label_core.cuh"

namespace rj {

LabelKernel label_points_count(int shape, int ni, int nf) { return label_kernel_cols<false>(shape, ni, nf); }

// Cell codes, one warp per cell of the (cnx + 1) x (cny + 1) map: the code
// its blocks share (a polygon, or none), else kCodeMixed.  Cell k of an axis
// holds the coordinates with k - 1/2 <= v * a + o <= k + 1/2; in tile c those
// lie at window coordinates h * (s * v + t) + h, off by at most `err` pixels
// in fp32.  A cell is uniform only when that range, widened by err, lies in
// one tile at least one pixel from its edges (no other tile's window then
// holds a point of the cell).
// The ranges are computed in fp32 (fp64 runs at a small fraction of its rate);
// err includes the rounding of that computation.
struct CellAxis {
    int lo, hi, tile;      // pixels of the tile; lo > hi: mixed
};
__device__ __forceinline__ CellAxis cell_axis(int k, float inv_a, float o, const TileAxis& x, float err) {
    const float v0 = ((float)k - 0.5f - o) * inv_a, v1 = ((float)k + 0.5f - o) * inv_a;
    CellAxis r{0, -1, 0};
    const float g = floorf((0.5f * (v0 + v1) - x.lb) * x.inv_td);
    if (!(g >= 0.0f && g < (float)x.split)) return r;
    r.tile = (int)g;
    const float4 f = __ldg(x.xf + r.tile);
    const float w0 = f.z * (f.x * v0 + f.y) + f.z - err;
    const float w1 = f.z * (f.x * v1 + f.y) + f.z + err;
    if (!(w0 >= 1.0f && w1 < (float)(x.res - 1))) return r;
    r.lo = (int)w0;
    r.hi = (int)w1;
    return r;
}

__global__ void k_label_cells(LabelPointArgs a, float ox, float oy, float errx, float erry, uint16_t* __restrict__ cells) {
    const int lane = threadIdx.x & 31;
    const int w = a.cnx + 1, total = w * (a.cny + 1);
    const float inv_ax = 1.0f / a.cax, inv_ay = 1.0f / a.cay;
    for (int s = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); s < total;
         s += (int)((gridDim.x * blockDim.x) >> 5)) {
        const int ky = s / w, kx = s - ky * w;
        if (kx == a.cnx || ky == a.cny) {   // past the grid
            if (lane == 0) cells[s] = kEmptyLabel;
            continue;
        }
        const CellAxis cx = cell_axis(kx, inv_ax, ox, a.ax, errx);
        const CellAxis cy = cell_axis(ky, inv_ay, oy, a.ay, erry);
        uint32_t code = kCodeMixed;
        if (cx.lo <= cx.hi && cy.lo <= cy.hi) {
            const int bx0 = cx.lo >> 4, bx1 = cx.hi >> 4, by0 = cy.lo >> 4, by1 = cy.hi >> 4;
            const uint32_t* c = a.tr.code + (size_t)(cy.tile * a.ax.split + cx.tile) * a.tr.bw * a.tr.bh;
            const uint32_t first = __ldg(c + by0 * a.tr.bw + bx0);
            bool same = first < (uint32_t)a.P || first == kTierEmpty;
            // lanes: two rows of 16 blocks at a time
            for (int bx = bx0 + (lane & 15); bx <= bx1; bx += 16)
                for (int by = by0 + (lane >> 4); by <= by1; by += 2) same &= __ldg(c + by * a.tr.bw + bx) == first;
            if (__all_sync(0xffffffffu, same)) code = first == kTierEmpty ? (uint32_t)kEmptyLabel : first;
        }
        if (lane == 0) cells[s] = (uint16_t)code;
    }
}

void launch_label_cells(const LabelPointArgs& a, float ox, float oy, float errx, float erry, uint16_t* cells, int sms,
                        cudaStream_t st) {
    const long long warps = (long long)(a.cnx + 1) * (a.cny + 1);
    const long long blocks = std::max(1LL, std::min((warps * 32 + 255) / 256, (long long)sms * 16));
    k_label_cells<<<(unsigned)blocks, 256, 0, st>>>(a, ox, oy, errx, erry, cells);
    ++g_kernel_launches;
}

namespace {

int g_label_optin = -1;

// histogram copies: a power of two up to the warps of the block, within 32 KB
int label_copies(int shape, int P, bool agg) {
    const size_t per = (size_t)P * (agg ? 3 : 1) * 4;
    int copies = 1;
    while (copies * 2 <= kLabelShapes[shape].block / 32 && per * copies * 2 <= 32 * 1024) copies *= 2;
    return copies;
}

}  // namespace

int label_shapes() { return kNumLabelShapes; }

size_t label_points_smem(int shape, int cell_words, int P, bool agg) {
    if (shape < 0 || shape >= kNumLabelShapes) return 0;
    const LabelShape& s = kLabelShapes[shape];
    const size_t queue = (size_t)(s.block / 32) * (32 + 64 * std::min(s.nv, 2)) * (agg ? 12 : 8);
    return 2 * kLeanMaxSplit * sizeof(float) + queue + (size_t)cell_words * 4 +
           (size_t)label_copies(shape, P, agg) * P * (agg ? 3 : 1) * 4;
}

// false: the shape cannot run this query (columns, shared memory); nothing launched
bool launch_label_points(int shape, const LabelPointArgs& a, const LeanCols& lc_in, int sms, cudaStream_t st) {
    if (shape < 0 || shape >= kNumLabelShapes || a.ax.split > kLeanMaxSplit || a.ay.split > kLeanMaxSplit) return false;
    const bool agg = lc_in.aggr != 0;
    const int ni = lc_in.nint, nf = lc_in.ncol - lc_in.nint;
    LabelKernel k = agg ? label_points_sum(shape, ni, nf) : label_points_count(shape, ni, nf);
    if (!k) return false;
    LeanCols lc = lc_in;
    lc.copies = label_copies(shape, a.P, agg);
    return launch_label_kernel(k, kLabelShapes[shape].block, kLabelShapes[shape].nv,
                               label_points_smem(shape, a.cell_words, a.P, agg), a, lc, sms, st);
}

bool launch_label_kernel(LabelKernel k, int block, int nv, size_t smem, const LabelPointArgs& a, const LeanCols& lc,
                         int sms, cudaStream_t st) {
    if (g_label_optin < 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_label_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    }
    if (smem > (size_t)g_label_optin) return false;
    if (allow_smem(reinterpret_cast<const void*>(k), smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, block, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    const uint64_t per_iter = (uint64_t)block * nv;
    const uint64_t need = ((a.n >> 1) + per_iter - 1) / per_iter;
    const uint64_t blocks = std::min<uint64_t>((uint64_t)sms * per_sm, std::max<uint64_t>(need, 1));
    // shared counts are 32-bit: a block must see fewer than 2^31 points (a
    // point on a seam counts up to four times)
    if (a.n / blocks >= (1ull << 29)) return false;
    k<<<(unsigned)blocks, block, smem, st>>>(a, lc);
    ++g_kernel_launches;
    return true;
}

}  // namespace rj
