// What the forward and backward blends share: the block size, the margin that
// covers the per-pixel test's rounding, and the conservative shapes made with
// it: a record's box (the backward's warps test it before they walk a record)
// and its cells of a tile (the forward's lists).
#pragma once

#include "raster_common.cuh"

namespace lrt {
namespace {

constexpr uint32_t kBlendThreads = 256;

// The float power of a pixel can fall below the exact one by at
// most ~4u (|a| dx^2 + 2|b| |dx dy| + |c| dy^2) <= 4u kappa power with
// kappa = (|a| + 2|b| + |c|) / lambda_min; det = a c - b^2 itself carries a
// relative error up to ~4u (|ac| + b^2) / det. delta bounds both with a factor
// of 8 to spare. False where it is not small (or the conic not one of an
// ellipse): such a record is never skipped. The divisions and roots are the hardware's approximate ones (a few 2^-22 of
// relative error; a quotient by more than 2^126 is excluded by the bound on
// the conic's trace): delta is at least 1.3e-5 and holds a factor of 8, so
// both bounds still hold.
__device__ __forceinline__ float approx_sqrt(float v) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ bool cut_margin(float a, float b, float c, float cutoff, float& det, float& invDet,
                                           float& delta) {
    det = a * c - b * b;
    const float half = 0.5f * (a + c);
    const float root = approx_sqrt(0.25f * (a - c) * (a - c) + b * b);
    // root's own error (a few 2^-22 of at most half) taken off lmin.
    const float lmin = half - root - 2.0e-6f * half;
    if (!(det > 0.0f) || !(lmin > 0.0f) || !(cutoff >= 0.0f) || !(half < 1.0e30f)) return false;
    invDet = __fdividef(1.0f, det);
    const float kappa = __fdividef(fabsf(a) + 2.0f * fabsf(b) + fabsf(c), lmin);
    const float cond = (fabsf(a * c) + b * b) * invDet;
    delta = 32.0f * 5.9604645e-08f * (kappa + cond + 4.0f);
    return delta < 0.25f;
}

// A box outside which no pixel centre can pass the record's cut, so that
// skipping a record for a whole warp never changes a pixel. {power <= k} is an
// ellipse whose bounding half-widths are sqrt(k c / det) and sqrt(k a / det)
// for the conic (a, b, c); the cut is widened to cutoff / (1 - delta) and the
// half-widths by (1 + delta) plus 1e-3 px.
__device__ __forceinline__ float4 cull_box(const ProjRecord& rec) {
    const float a = rec.conic.x, b = rec.conic.y, c = rec.conic.z, cutoff = rec.screen.w;
    const float kInf = 3.0e38f;
    float det, invDet, delta;
    if (!cut_margin(a, b, c, cutoff, det, invDet, delta)) return make_float4(-kInf, kInf, -kInf, kInf);
    const float k = __fdividef(cutoff, 1.0f - delta) * invDet;
    const float ex = approx_sqrt(k * c) * (1.0f + delta) + 1e-3f;
    const float ey = approx_sqrt(k * a) * (1.0f + delta) + 1e-3f;
    if (!(ex < kInf) || !(ey < kInf)) return make_float4(-kInf, kInf, -kInf, kInf);
    return make_float4(rec.screen.x - ex, rec.screen.x + ex, rec.screen.y - ey, rec.screen.y + ey);
}

// The tile's 16 cells of 4x4 pixels, cell 4 r + c at row r, column c.
constexpr uint32_t kCells = 16;

// The cells of the tile at pixel (x0, y0) where a pixel may pass the record's
// cut, a bit each (the rest certainly hold none). Over a band of rows
// dy in [lo, hi] the ellipse {power <= k} spans, on its right,
// x(dy) = (-b dy + sqrt(k a - det dy^2)) / a, which rises to the ellipse's
// rightmost point (dy = -b ex / c) and falls past it, so its largest value
// over the band is at that dy clamped into the band; the left side mirrors
// it. k is cull_box's widened cut, widened by another 4 delta: delta bounds
// det's relative error and is at least 1.3e-5, so k a - det dy^2 as computed
// is not below the exact one; what is left, the rounding of the two terms
// and of their sum, is below 1e-5 of the extents. Measured on 1M splats,
// 1080p, the ellipse leaves 20% fewer (cell, record) steps than its
// bounding box.
__device__ __forceinline__ uint32_t cells_touched(const ProjRecord& rec, float x0, float y0) {
    const float a = rec.conic.x, b = rec.conic.y, c = rec.conic.z, cutoff = rec.screen.w;
    float det, invDet, delta;
    if (!cut_margin(a, b, c, cutoff, det, invDet, delta)) return 0xFFFFu;
    const float k = __fdividef(cutoff, 1.0f - delta) * (1.0f + 4.0f * delta);
    const float ex = approx_sqrt(k * invDet * c) * (1.0f + delta) + 1e-3f;
    const float ey = approx_sqrt(k * invDet * a) * (1.0f + delta) + 1e-3f;
    if (!(ex < 1.0e6f) || !(ey < 1.0e6f)) return 0xFFFFu;
    const float invA = __fdividef(1.0f, a);
    const float tip = -b * __fdividef(ex, c);   // dy of the rightmost point
    const float ka = k * a;
    const float slack = 1e-3f + 1e-5f * ex;
    const float cx = rec.screen.x - x0 - 0.5f, cy = rec.screen.y - y0 - 0.5f;   // from the tile's first pixel centre
    uint32_t cells = 0;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const float lo = 4.0f * static_cast<float>(r) - cy, hi = lo + 3.0f;
        const float yr = fminf(fmaxf(tip, lo), hi), yl = fminf(fmaxf(-tip, lo), hi);
        const float xr = (approx_sqrt(fmaxf(ka - det * yr * yr, 0.0f)) - b * yr) * invA + slack + cx;
        const float xl = (-approx_sqrt(fmaxf(ka - det * yl * yl, 0.0f)) - b * yl) * invA - slack + cx;
        // Column k's pixel centres are 4 k .. 4 k + 3: touched when
        // xl <= 4 k + 3 and xr >= 4 k.
        uint32_t row = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
            if (!(xl > 4.0f * static_cast<float>(q) + 3.0f) && !(xr < 4.0f * static_cast<float>(q))) row |= 1u << q;
        if (!(lo > ey) && !(hi < -ey)) cells |= row << (4 * r);
    }
    return cells;
}

}  // namespace
}  // namespace lrt
