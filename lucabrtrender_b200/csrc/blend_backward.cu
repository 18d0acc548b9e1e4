// The backward of the training blend (blend_kernel<true>): per pixel the
// forward's loop run backwards, gradients per pair summed without atomics.
//
// This file is compiled with fused multiply-add contraction allowed: its
// results are checked against FP64 oracles to a tolerance, not bit for bit,
// and every decision it shares with the forward (the power against the cut,
// alpha against 1/255 and 0.99) is computed by the same explicit
// expressions as there (splat_power's fused multiply-adds, lrt_exp near the
// thresholds), which contraction leaves unchanged.
#include "kernels.cuh"
#include "raster_common.cuh"
#include "blend_common.cuh"

namespace lrt {
namespace {

// d/du of the sRGB-to-linear curve (color.slang:7-10): 0 below zero, 1/12.92
// on the linear segment, 2.4/1.055 ((u + 0.055)/1.055)^1.4 above it.
__device__ __forceinline__ float srgb_to_linear_slope(float c) {
    if (!(c > 0.0f)) return 0.0f;
    if (c <= 0.04045f) return 1.0f / 12.92f;
    return 2.4f / 1.055f * lrt_pow((c + 0.055f) / 1.055f, 1.4f);
}

// Per pair, as written: d/d(centre x, centre y, conic a, b, c, alpha, r, g,
// b). While a batch is summed, with ga = dL/dalpha alpha (0 where alpha is
// clamped), slots 0..4 hold the sums of ga dx, ga dy, ga dx^2, ga dx dy and
// ga dy^2 and slot 5 that of ga: dL/dpower = -ga / 2 and dL/dalpha0 = ga /
// alpha0, so the record's alpha0, its conic and the factors are applied once,
// when the partials are written.
constexpr uint32_t kGrads = 9;
constexpr uint32_t kGradStride = 12;   // floats per pair in the partials buffer (three 16-byte vectors)
constexpr uint32_t kBwdPix = 4;        // pixels a thread: a column of its cell
constexpr uint32_t kBwdThreads = kBlendThreads / kBwdPix;
constexpr uint32_t kBwdBatch = 32;     // records a batch: a cell's four threads list eight each
constexpr uint32_t kCellThreads = 4;

struct BackwardShared {
    __align__(16) ProjRecord rec[kBwdBatch];    // the batch arriving
    __align__(16) ProjRecord walk[kBwdBatch];   // the batch being walked, last pair first
    // A record's cells (cells_touched, without the cells whose pixels all
    // stopped before it): record 8 g + 4 h + k in half h of word 4 g + k.
    __align__(16) uint16_t touched[kBwdBatch];
    uint8_t list[kCells][kBwdBatch];            // per cell its records' indices, last pair first
    uint32_t emit[kBwdBatch];
    uint32_t cellLast[kCells];                  // one past the last pair any of the cell's pixels took
    float part[kCells][kBwdBatch][kGrads];
};
__device__ __forceinline__ float2 twice(float v) { return make_float2(v, v); }
__device__ __forceinline__ float& half_of(float2& v, uint32_t k) { return (k & 1u) == 0 ? v.x : v.y; }
__device__ __forceinline__ float half_of(const float2& v, uint32_t k) { return (k & 1u) == 0 ? v.x : v.y; }
__device__ __forceinline__ uint32_t touched_place(uint32_t m) {
    return (m & ~7u) + 2u * (m & 3u) + ((m >> 2) & 1u);
}

// Sum of nine values over a cell's four lanes by recursive halving (a
// reduce-scatter): at each step a lane keeps part of its list, sends the rest
// to its partner and adds what it receives. The list shrinks 9 -> 5 -> 3
// (lists padded with zeros where a half is shorter), so 5 + 3 shuffles
// replace 9 x 2 butterflies. Lane l then holds the sums of values
// 5 l2 + 3 l1 and the two after it (l2, l1: its bits), as far as they are in
// its list.
__device__ __forceinline__ float3 cell_reduce_scatter9(const float (&v)[9], bool u2, bool u1) {
    constexpr unsigned kAll = 0xFFFFFFFFu;
    float a[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {   // [0..4] | [5..8, -]
        const float lo = v[j], hi = j < 4 ? v[5 + j] : 0.0f;
        a[j] = (u2 ? hi : lo) + __shfl_xor_sync(kAll, u2 ? lo : hi, 2);
    }
    float b[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {   // [0, 1, 2] | [3, 4, -]
        const float lo = a[j], hi = j < 2 ? a[3 + j] : 0.0f;
        b[j] = (u1 ? hi : lo) + __shfl_xor_sync(kAll, u1 ? lo : hi, 1);
    }
    return make_float3(b[0], b[1], b[2]);
}

// The backward of blend_kernel<true>: per pixel, the reference's loop run
// backwards from the last pair that contributed, rebuilding each pair's
// transmittance from the final one (T_i = T_{i+1} / (1 - alpha_i)) rather
// than storing it, with B the colour behind the pair:
//   dL/dc_i     = dL/drgb * T_i alpha_i
//   dL/dalpha_i = T_i sum_k dL/drgb_k (c_ik - B_k) - dL/dT * T / (1 - alpha_i)
//   B          <- alpha_i c_i + (1 - alpha_i) B
// then through alpha = min(0.99, alpha0 exp(-power / 2)) (no gradient when
// clamped) and power = a dx^2 + 2 b dx dy + c dy^2.
//
// Bound by instruction issue. As in the forward, each 4x4 cell of the tile
// walks its own list of the batch's records (four pixels a thread, a cell's
// four lanes side by side with the warp's seven other cells), so that a
// step's work is spent on pixels the records reach, and the sum of a pair's
// nine values over pixels takes two halving steps over a cell's four lanes
// for eight records at once. Each (cell, record) sum has a place of its
// own in shared memory; after the walk they are added in cell order and
// written at the pair's emit index: no atomics, and the sums are the same
// every time. A splat's pairs are contiguous there, so its sum needs none
// either. Batches of 32 keep those sums at 18 KB a block, ten blocks an SM.
// 1M splats at 1080p: 0.742 ms with 8x8 blocks visiting records, 0.790 with
// two pixels a thread, batches of 64 and a branch a pixel, 0.709 with four
// pixels and 32, 0.605 without the branches (four independent chains a lane;
// 61% of the issue slots and 14% second slots of packed operations). Bounds
// of 9 and 12 blocks an SM: 0.623 and 0.640.
// One tile: `item` indexes the ranges (the frame's tile, or a batch's
// (view, tile) item); (tx, ty) is the tile within its view.
__device__ __forceinline__ void blend_backward_tile(const BlendParams& bp, uint32_t item, uint32_t tx, uint32_t ty,
                                                    const uint2* __restrict__ ranges,
                                                    const unsigned long long* __restrict__ pairs,
                                                    const uint32_t* __restrict__ emit,
                                                    const uint32_t* __restrict__ emitSlot,
                                                    const ProjRecord* __restrict__ proj,
                                                    const float4* __restrict__ pixState,
                                                    const uint32_t* __restrict__ pixLast,
                                                    const float4* __restrict__ gradColour,
                                                    float* __restrict__ partials) {
    constexpr uint32_t kP = kBwdPix;
    __shared__ BackwardShared sh;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    // Warp w holds cells 8 w .. 8 w + 7, four lanes each, a lane a column of its cell.
    const uint32_t cell = warp * 8u + (lane >> 2);
    const uint32_t px = tx * kTile + (cell & 3u) * 4u + (lane & 3u);
    const uint32_t py0 = ty * kTile + (cell >> 2) * 4u;
    const uint2 range = ranges[item];
    const uint32_t start = range.x;
    const uint32_t slotMask = static_cast<uint32_t>((1ull << bp.slotBits) - 1ull);
    auto lowWord = [&](uint32_t k) {   // a pair word's low field, or the slot alone
        return __ldg(reinterpret_cast<const uint32_t*>(pairs) + (static_cast<size_t>(k) << bp.pairShift)) & slotMask;
    };
    const float pxf = static_cast<float>(px) + 0.5f;
    const float tileX = static_cast<float>(tx * kTile), tileY = static_cast<float>(ty * kTile);

    // The lane's four pixels, a column of its cell, as two pairs: pixel
    // 2 h + k is half k of pair h.
    uint32_t myLast[kP];
    float2 py[kP / 2], gr[kP / 2], gg[kP / 2], gb[kP / 2], T[kP / 2], gTT[kP / 2], Br[kP / 2], Bg[kP / 2], Bb[kP / 2];
    uint32_t laneMax = start;
    bool unusual = false;   // a pixel's gradient is not finite
#pragma unroll
    for (uint32_t q = 0; q < kP; ++q) {
        const uint32_t row = py0 + q;
        const bool inside = px < bp.width && row < bp.height;
        myLast[q] = start;
        float r = 0.0f, g = 0.0f, b = 0.0f, t = 1.0f, gT = 0.0f;
        if (inside) {
            const size_t pix = static_cast<size_t>(row) * bp.width + px;
            myLast[q] = pixLast[pix];
            const float4 st = pixState[pix];
            const float4 G = gradColour[pix];
            t = st.w;
            const float cov = 1.0f - t;
            if (bp.linearise != 0 && cov > 1e-6f) {
                const float u0 = st.x / cov, u1 = st.y / cov, u2 = st.z / cov;
                const float d0 = srgb_to_linear_slope(u0), d1 = srgb_to_linear_slope(u1), d2 = srgb_to_linear_slope(u2);
                r = G.x * d0;
                g = G.y * d1;
                b = G.z * d2;
                // out_k = s(u_k) cov + T bg_k with cov = 1 - T; alpha_out = cov + T bg_a
                gT = G.x * (bp.bg[0] - (srgb_to_linear(u0) - d0 * u0)) +
                     G.y * (bp.bg[1] - (srgb_to_linear(u1) - d1 * u1)) +
                     G.z * (bp.bg[2] - (srgb_to_linear(u2) - d2 * u2)) + G.w * (bp.bg[3] - 1.0f);
            } else {
                r = G.x;
                g = G.y;
                b = G.z;
                gT = G.x * bp.bg[0] + G.y * bp.bg[1] + G.z * bp.bg[2] + G.w * (bp.bg[3] - 1.0f);
            }
        }
        half_of(py[q / 2], q) = static_cast<float>(row) + 0.5f;
        half_of(gr[q / 2], q) = r;
        half_of(gg[q / 2], q) = g;
        half_of(gb[q / 2], q) = b;
        half_of(T[q / 2], q) = t;
        half_of(gTT[q / 2], q) = -gT * t;   // the final transmittance's share of every dL/dalpha
        half_of(Br[q / 2], q) = 0.0f;
        half_of(Bg[q / 2], q) = 0.0f;
        half_of(Bb[q / 2], q) = 0.0f;
        unusual = unusual || !(finite(r) && finite(g) && finite(b) && finite(gT));
        laneMax = max(laneMax, myLast[q]);
    }
    {
        uint32_t most = laneMax;
#pragma unroll
        for (uint32_t d = 1; d < kCellThreads; d <<= 1) most = max(most, __shfl_xor_sync(0xFFFFFFFFu, most, d));
        if ((lane & (kCellThreads - 1u)) == 0) sh.cellLast[cell] = most;
    }
    const bool pixelsFinite = __syncthreads_or(unusual ? 1 : 0) == 0;
    uint32_t maxLast = start;
#pragma unroll
    for (uint32_t q = 0; q < kCells; ++q) maxLast = max(maxLast, sh.cellLast[q]);
    // Pairs past every pixel's last contributor get zero partials here, so the
    // buffer needs no clearing beforehand.
    for (uint32_t k = maxLast + tid; k < range.y; k += kBwdThreads) {
        const uint32_t e = emitSlot != nullptr ? lowWord(k) : emit[k];
        float4* out = reinterpret_cast<float4*>(partials + static_cast<size_t>(e) * kGradStride);
        out[0] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        out[1] = out[0];
        out[2] = out[0];
    }

    // A batch's record m is pair bEnd - 1 - m. Its slot and emit index: the
    // emit index is the word's low field (and the slot comes from the
    // emit-slot map), or it travelled through the sort as a value.
    uint32_t nextSlot = 0, nextEmit = 0;
    auto fetch_index = [&](uint32_t end) {
        if (tid >= kBwdBatch || end <= start || tid >= end - start) return;
        const uint32_t at = end - 1u - tid;
        const uint32_t low = lowWord(at);
        nextSlot = emitSlot != nullptr ? emitSlot[low] : low;
        nextEmit = emitSlot != nullptr ? low : emit[at];
    };
    auto fetch_record = [&](uint32_t end) {
        if (tid >= kBwdBatch || end <= start || tid >= end - start) return;
        const float4* src = reinterpret_cast<const float4*>(proj + nextSlot);
        float4* dst = reinterpret_cast<float4*>(&sh.rec[tid]);
#pragma unroll
        for (int q = 0; q < 3; ++q) cp_async16(dst + q, src + q);
    };
    // Where the lane's three sums of a reduce-scatter go, and which it has (always the first).
    const bool u2 = (lane & 2u) != 0, u1 = (lane & 1u) != 0;
    const uint32_t sumAt = (u2 ? 5u : 0u) + (u1 ? 3u : 0u);
    const bool has1 = !(u2 && u1), has2 = !u1;

    fetch_index(maxLast);
    fetch_record(maxLast);
    for (uint32_t bEnd = maxLast; bEnd > start;) {
        const uint32_t cnt = min(bEnd - start, kBwdBatch);
        const uint32_t bStart = bEnd - cnt;
        bool oddRecord = false;   // its colour is not finite
        if (tid < kBwdBatch) {
            uint32_t touched = 0;
            if (tid < cnt) {
                cp_async_wait_all();
                const ProjRecord rec = sh.rec[tid];
                sh.walk[tid] = rec;
                sh.emit[tid] = nextEmit;
                oddRecord = !(finite(rec.colour.x) && finite(rec.colour.y) && finite(rec.colour.z));
                touched = cells_touched(rec, tileX, tileY);
#pragma unroll
                for (uint32_t q = 0; q < kCells; ++q)
                    if (sh.cellLast[q] <= bEnd - 1u - tid) touched &= ~(1u << q);
            }
            sh.touched[touched_place(tid)] = static_cast<uint16_t>(touched);
            fetch_index(bStart);
        }
        const bool allFinite = __syncthreads_or(oddRecord ? 1 : 0) == 0 && pixelsFinite;
        fetch_record(bStart);
        uint32_t count;
        {
            const uint32_t part = lane & (kCellThreads - 1u);
            const uint4 marks = *reinterpret_cast<const uint4*>(&sh.touched[8u * part]);
            const uint32_t word[4] = {marks.x, marks.y, marks.z, marks.w};
            uint32_t bits = 0;   // bits k and 16 + k: records k and 4 + k
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) bits |= ((word[k] >> cell) & 0x00010001u) << k;
            bits = (bits | bits >> 12) & 0xFFu;
            const uint32_t own = static_cast<uint32_t>(__popc(bits));
            uint32_t upTo = own;
#pragma unroll
            for (uint32_t d = 1; d < kCellThreads; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, upTo, d, kCellThreads);
                if (part >= d) upTo += o;
            }
            count = __shfl_sync(0xFFFFFFFFu, upTo, kCellThreads - 1u, kCellThreads);
            uint8_t* at = &sh.list[cell][upTo - own];
            for (; bits != 0; bits &= bits - 1u) *at++ = static_cast<uint8_t>(8u * part + __ffs(bits) - 1u);
            __syncwarp();
        }
        for (uint32_t i = 0; __any_sync(0xFFFFFFFFu, i < count); ++i) {
            const bool mine = i < count;
            const uint32_t j = mine ? sh.list[cell][i] : 0u;
            const ProjRecord rec = sh.walk[j];
            const uint32_t at = mine ? bEnd - 1u - j : 0xFFFFFFFFu;   // the pair (none: past every pixel's last)
            // splat_power's operations, a pair of pixels at a time.
            const float dx = pxf - rec.screen.x;
            const float t = rec.conic.x * dx * dx, u = 2.0f * rec.conic.y * dx;
            float v[kGrads] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            float sum = 0.0f, sumY = 0.0f, sumYY = 0.0f;   // of ga, ga dy and ga dy^2: dx is the lane's
            bool hitAny = false;
#pragma unroll
            for (uint32_t h = 0; h < kP / 2; ++h) {
                const float2 dy = __fadd2_rn(py[h], twice(-rec.screen.y));
                const float2 power =
                    __ffma2_rn(__fmul2_rn(twice(rec.conic.z), dy), dy, __ffma2_rn(twice(u), dy, twice(t)));
                // The forward's alpha, so the same pixels took the record.
                const float2 raw = lrt_scaled_exp_half2(rec.conic.w, power);
                const float a0 = fminf(0.99f, raw.x), a1 = fminf(0.99f, raw.y);
                const bool take0 = at < myLast[2 * h] && !(power.x > rec.screen.w) && !(a0 < 1.0f / 255.0f);
                const bool take1 = at < myLast[2 * h + 1] && !(power.y > rec.screen.w) && !(a1 < 1.0f / 255.0f);
                hitAny = hitAny || take0 || take1;
                // A pixel that did not take the record goes through the same
                // steps with alpha 0: they change nothing while all that
                // enters them is finite, and where something is not, its
                // results are dropped.
                const float2 alpha = make_float2(take0 ? a0 : 0.0f, take1 ? a1 : 0.0f);
                const float2 open = __ffma2_rn(alpha, twice(-1.0f), twice(1.0f));   // 1 - alpha, in [0.01, 1]
                float2 inv;   // 1 / (1 - alpha) to about 1 ulp
                asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.x) : "f"(open.x));
                asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.y) : "f"(open.y));
                const float2 Ti = __fmul2_rn(T[h], inv);
                const float2 w = __fmul2_rn(Ti, alpha);
                const float2 cr = __ffma2_rn(Br[h], twice(-1.0f), twice(rec.colour.x));
                const float2 cg = __ffma2_rn(Bg[h], twice(-1.0f), twice(rec.colour.y));
                const float2 cb = __ffma2_rn(Bb[h], twice(-1.0f), twice(rec.colour.z));
                const float2 behind = __ffma2_rn(gr[h], cr, __ffma2_rn(gg[h], cg, __fmul2_rn(gb[h], cb)));
                const float2 dAlpha = __ffma2_rn(Ti, behind, __fmul2_rn(gTT[h], inv));
                float2 ga = make_float2(raw.x <= 0.99f ? alpha.x : 0.0f, raw.y <= 0.99f ? alpha.y : 0.0f);
                ga = __fmul2_rn(dAlpha, ga);
                if (allFinite) {
                    v[6] = __fmaf_rn(gr[h].x, w.x, __fmaf_rn(gr[h].y, w.y, v[6]));
                    v[7] = __fmaf_rn(gg[h].x, w.x, __fmaf_rn(gg[h].y, w.y, v[7]));
                    v[8] = __fmaf_rn(gb[h].x, w.x, __fmaf_rn(gb[h].y, w.y, v[8]));
                    Br[h] = __ffma2_rn(alpha, cr, Br[h]);
                    Bg[h] = __ffma2_rn(alpha, cg, Bg[h]);
                    Bb[h] = __ffma2_rn(alpha, cb, Bb[h]);
                    T[h] = Ti;
                } else {
#pragma unroll
                    for (uint32_t k = 0; k < 2; ++k) {
                        if (!(k == 0 ? take0 : take1)) {
                            half_of(ga, k) = 0.0f;
                            continue;
                        }
                        if (!(half_of(raw, k) <= 0.99f)) half_of(ga, k) = 0.0f;
                        v[6] += half_of(gr[h], k) * half_of(w, k);
                        v[7] += half_of(gg[h], k) * half_of(w, k);
                        v[8] += half_of(gb[h], k) * half_of(w, k);
                        half_of(Br[h], k) = __fmaf_rn(half_of(alpha, k), half_of(cr, k), half_of(Br[h], k));
                        half_of(Bg[h], k) = __fmaf_rn(half_of(alpha, k), half_of(cg, k), half_of(Bg[h], k));
                        half_of(Bb[h], k) = __fmaf_rn(half_of(alpha, k), half_of(cb, k), half_of(Bb[h], k));
                        half_of(T[h], k) = half_of(Ti, k);
                    }
                }
                const float2 gy = __fmul2_rn(ga, dy);
                sum += ga.x + ga.y;
                sumY += gy.x + gy.y;
                sumYY = __fmaf_rn(gy.x, dy.x, __fmaf_rn(gy.y, dy.y, sumYY));
            }
            v[0] = sum * dx;
            v[1] = sumY;
            v[2] = v[0] * dx;
            v[3] = sumY * dx;
            v[4] = sumYY;
            v[5] = sum;
            float3 sums = make_float3(0.0f, 0.0f, 0.0f);
            if (__any_sync(0xFFFFFFFFu, hitAny)) sums = cell_reduce_scatter9(v, u2, u1);
            if (mine) {
                float* out = &sh.part[cell][j][sumAt];
                out[0] = sums.x;
                if (has1) out[1] = sums.y;
                if (has2) out[2] = sums.z;
            }
        }
        __syncthreads();
        // Two threads a record: its sums over the cells it reached, in cell
        // order; the first writes slots 0..3, the second the rest.
        const uint32_t m = tid >> 1;
        if (m < cnt) {
            const bool second = (tid & 1u) != 0;
            uint32_t cells = sh.touched[touched_place(m)];
            float sum[5] = {0, 0, 0, 0, 0};
            for (; cells != 0; cells &= cells - 1u) {
                const float* src = sh.part[__ffs(cells) - 1][m] + (second ? 4 : 0);
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) sum[k] += src[k];
                if (second) sum[4] += src[4];
            }
            const float4 conic = sh.walk[m].conic;
            float4* out = reinterpret_cast<float4*>(partials + static_cast<size_t>(sh.emit[m]) * kGradStride);
            if (!second) {
                const float gx = __fmaf_rn(conic.x, sum[0], conic.y * sum[1]);
                const float gy = __fmaf_rn(conic.y, sum[0], conic.z * sum[1]);
                out[0] = make_float4(gx, gy, -0.5f * sum[2], -sum[3]);
            } else {
                out[1] = make_float4(-0.5f * sum[0], sum[1] / conic.w, sum[2], sum[3]);
                out[2] = make_float4(sum[4], 0.0f, 0.0f, 0.0f);
            }
        }
        __syncthreads();
        bEnd = bStart;
    }
}

template <bool kChained>
__global__ void __launch_bounds__(kBwdThreads)
blend_backward_kernel(BlendParams bp, const uint2* __restrict__ ranges, const unsigned long long* __restrict__ pairs,
                      const uint32_t* __restrict__ emit, const uint32_t* __restrict__ emitSlot,
                      const ProjRecord* __restrict__ proj,
                      const float4* __restrict__ pixState, const uint32_t* __restrict__ pixLast,
                      const float4* __restrict__ gradColour, float* __restrict__ partials,
                      const uint32_t* __restrict__ order) {
    chained_entry<kChained>();
    const uint32_t tile = order != nullptr ? order[blockIdx.x] : blockIdx.x;
    blend_backward_tile(bp, tile, tile % bp.tilesX, tile / bp.tilesX, ranges, pairs, emit, emitSlot, proj, pixState,
                        pixLast, gradColour, partials);
}

// The backward of a training batch: one block per (view, tile) item of the
// chunk, each the tile of blend_backward_kernel in its own view (records at
// the view's base, pixel state and colour gradient from the view's buffers).
__global__ void __launch_bounds__(kBwdThreads)
blend_backward_batch_kernel(BlendParams bp, const ViewParams* __restrict__ views, uint32_t viewCount,
                            const uint2* __restrict__ ranges, const unsigned long long* __restrict__ pairs,
                            const uint32_t* __restrict__ emit, const ProjRecord* __restrict__ proj,
                            float* __restrict__ partials) {
    const uint32_t item = blockIdx.x;
    uint32_t lo = 0, hi = viewCount;   // the view whose tiles hold `item`
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (views[mid].tileBase <= item) lo = mid; else hi = mid;
    }
    const ViewParams v = views[lo];
    BlendParams vbp = bp;
    vbp.width = v.width;
    vbp.height = v.height;
    vbp.tilesX = v.tilesX;
    const uint32_t local = item - v.tileBase;
    blend_backward_tile(vbp, item, local % v.tilesX, local / v.tilesX, ranges, pairs, emit, nullptr,
                        proj + v.recordBase, v.pixState, v.pixLast, v.gradColour, partials);
}

}  // namespace

cudaError_t launch_blend_backward_batch(const BlendParams& bp, const ViewParams* views, uint32_t viewCount,
                                        const uint2* ranges, const uint64_t* pairs, const uint32_t* emit,
                                        const ProjRecord* proj, uint32_t totalTiles, float* partials,
                                        cudaStream_t stream) {
    if (totalTiles == 0) return cudaSuccess;
    blend_backward_batch_kernel<<<totalTiles, kBwdThreads, 0, stream>>>(
        bp, views, viewCount, ranges, reinterpret_cast<const unsigned long long*>(pairs), emit, proj, partials);
    return cudaGetLastError();
}

cudaError_t launch_blend_backward(const BlendParams& bp, const uint2* ranges, const uint64_t* pairs,
                                  const uint32_t* emit, const uint32_t* emitSlot, const ProjRecord* proj,
                                  const float4* pixState, const uint32_t* pixLast, const float4* gradColour,
                                  float* partials, cudaStream_t stream, const uint32_t* order) {
    const uint32_t tiles = bp.tilesX * bp.tilesY;
    if (tiles == 0) return cudaSuccess;
    return launch_chained(blend_backward_kernel<true>, blend_backward_kernel<false>, dim3(tiles), dim3(kBwdThreads), 0, stream, bp, ranges,
                          reinterpret_cast<const unsigned long long*>(pairs), emit, emitSlot, proj, pixState, pixLast,
                          gradColour, partials, order);
}

}  // namespace lrt
