// rj_lean.cuh -- building blocks of the lean point passes: the mixed-code
// marker and the pixel arithmetic.
#pragma once
#include "rj_launch.h"

namespace rj {

// Marker in a block-code map: the block's pixels carry different labels.
// 0xFFFD is no polygon label (ids stop at kMaxLabelPolys - 1), nor the empty
// or the hybrid border label.
constexpr uint16_t kCodeMixed = 0xFFFDu;

// Pixel of (x, y) in the tile, equal to pix_of(snap_win(win_coord(...))) of
// the generic pass with fewer operations, by two exact rewrites:
//   * the snap's multiplication by 256 moves into the viewport transform:
//     fl(fl(h*ndc) + h) * 256 == fl(fl(H*ndc) + H) with H = 256 h, since
//     scaling by a power of two commutes with rounding (an h*ndc small enough
//     to be subnormal is absorbed by the addition of h either way);
//   * snap_win clamps the window coordinate to +-2^20 px before converting;
//     here only the lower clamp stays (it also sends NaN below the canvas:
//     fmaxf(NaN, c) = c) and the conversion saturates above, which puts every
//     coordinate beyond the clamp on a pixel outside [0, res) just the same.
// (Packed fp32x2 arithmetic was tried for the two coordinates: each packed
// operation alone rounds like the scalar one, but chains of them did not
// reproduce the scalar results on GB300, so the arithmetic stays scalar.)
__device__ __forceinline__ int snapped_pixel(float v, float s, float t, float H) {
    const float w = __fadd_rn(__fmul_rn(H, __fadd_rn(__fmul_rn(s, v), t)), H);   // window coordinate * 256
    return __float2int_rn(fmaxf(w, -kWinClamp * (float)kSub)) >> kSubpixelBits;
}

}  // namespace rj
