// Stages (d) tile ranges and (e) the front-to-back blend.
//
// Pair words (64 bits, sorted on their tile bits, or on tile and depth):
//   single frames:  tile << 32 | slot (or emit index), emitted in depth order
//                   and sorted stably on the tile bits -- the reference's
//                   depth sort followed by a stable tile sort
//                   (shaders/lrt/splat/frame.slang:17-20,
//                   modules/render/src/TileRasterizer.cpp:401-457);
//   batched views:  tile << (24 + slotBits) | depthKey24 << slotBits | slot,
//                   emitted in slot order and sorted stably on the key bits.
// Both leave every tile's pairs in (depth key, slot) order. BlendParams
// carries the slot field's width (slotBits) and the tile field's shift.
#include "kernels.cuh"
#include "raster_common.cuh"
#include "blend_common.cuh"

namespace lrt {
namespace {

constexpr uint32_t kWaitLimit = 1u << 22;
// Pixels a thread in the blends, and the records a batch holds: one a thread.
constexpr uint32_t kBlendPix = 2;
constexpr uint32_t kBatch = kBlendThreads / kBlendPix;

// shaders/lrt/splat/splat_ranges.slang:11-25 (after a zeroing memset,
// splat_tiles_clear.slang:8-17). Each thread takes kRangeRun consecutive
// pairs (two 16-byte loads per pair pair) and the one before them.
constexpr uint32_t kRangeRun = 8;
template <bool kChained>
__global__ void ranges_kernel(const unsigned long long* __restrict__ pairs, const uint32_t* __restrict__ dCount,
                              uint32_t cap, uint32_t tileShift, uint2* __restrict__ ranges) {
    chained_entry<kChained>();
    const uint32_t n = min(*dCount, cap);
    const uint32_t first = (blockIdx.x * blockDim.x + threadIdx.x) * kRangeRun;
    if (first >= n) return;
    uint32_t prev = first == 0 ? 0xFFFFFFFFu : static_cast<uint32_t>(__ldg(pairs + first - 1) >> tileShift);
    unsigned long long w[kRangeRun];
    if (first + kRangeRun <= n) {
        const ulonglong2* v = reinterpret_cast<const ulonglong2*>(pairs + first);
#pragma unroll
        for (uint32_t k = 0; k < kRangeRun / 2; ++k) {
            const ulonglong2 q = __ldg(v + k);
            w[2 * k] = q.x;
            w[2 * k + 1] = q.y;
        }
    } else {
#pragma unroll
        for (uint32_t k = 0; k < kRangeRun; ++k) w[k] = first + k < n ? __ldg(pairs + first + k) : 0ull;
    }
#pragma unroll
    for (uint32_t k = 0; k < kRangeRun; ++k) {
        const uint32_t i = first + k;
        if (i < n) {
            const uint32_t t = static_cast<uint32_t>(w[k] >> tileShift);
            if (t != prev) {
                ranges[t].x = i;
                if (i > 0) ranges[prev].y = i;
            }
            prev = t;
        }
    }
    // The run's last pair closes its tile when the pair after it (or the end) differs.
    const uint32_t last = min(first + kRangeRun, n) - 1;
    if (last + 1 == n || static_cast<uint32_t>(__ldg(pairs + last + 1) >> tileShift) != prev) ranges[prev].y = last + 1;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// One record (48 bytes, 16-byte aligned at both ends) by the bulk-copy engine.
__device__ __forceinline__ void bulk_copy_record(void* dst, const void* src, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 48, [%2];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Bounded wait on a barrier phase; false when the limit passed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    for (uint32_t it = 0; it < kWaitLimit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Eight threads own a cell of the tile, two pixels each (two rows apart).
constexpr uint32_t kCellThreads = 8;

// A record as the walk reads it: every factor twice, so that a 16-byte load
// gives two operands of the packed (two pixels at once) arithmetic.
struct __align__(16) PairRecord {
    float4 centre;   // -x, -x, -y, -y
    float4 ab;       // a, a, 2 b, 2 b
    float4 c;        // c, c, cutoff, alpha (a disc of a composite frame: -1)
    float4 rg;       // r, r, g, g
    float4 bz;       // b, b, view z, view z
};

struct BlendShared {
    __align__(128) ProjRecord rec[kBatch];    // the batch arriving
    PairRecord walk[kBatch + 1];              // the batch being walked, and one no pixel takes
    // A record's cells (cells_touched): record 16 g + 8 h + k in half h of
    // word 8 g + k.
    __align__(16) uint16_t touched[kBatch];
    // Per cell its records' indices in order, then up to three of the record
    // no pixel takes.
    __align__(16) uint8_t list[kCells][kBatch + 4];
    uint64_t bar;
};
static_assert(kBatch == 128 && kBatch == kCells * kCellThreads, "a thread lists 16 records of its cell");
struct CompositeShared {
    float zMax[kBatch];
    float warpMax[kBatch / 32];
};

__device__ __forceinline__ float2 lower2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 upper2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ bool finite(float v) { return fabsf(v) < INFINITY; }

// shaders/lrt/splat/splat_blend.slang:23-108 (splat-only entry, :110-114).
// One block of 128 threads per 16x16 tile, two pixels a thread. The tile's
// pairs are read in batches of 128, one record a thread, each copied into
// shared memory by a bulk copy completing on the block's mbarrier; a thread
// then writes its record out for the walk, so batch k+1 arrives in the same
// place while batch k is walked, and the pair words of batch k+2 are on their
// way in a register.
//
// The walk is bound by instruction issue and by the FMA pipe, which a packed
// operation holds for two cycles (1M splats at 1080p: 78% of the issue slots,
// 55% of the pipe; its records come from L2 and shared memory), and a splat of
// the usual size covers a third of the pixels of the 8x8 blocks it touches.
// So each 4x4 cell walks its own list: a thread marks the cells its record may
// touch (cells_touched), and each cell's eight threads read 16 records' marks
// each and write the indices of those that may touch it, in order. A warp
// walks the lists of its four cells side by side and takes as many steps as
// its longest list has records. A lane's two pixels go through a step together
// in packed single precision, each operation one instruction for both and
// rounded as the scalar one is, and two records' powers and alphas are formed
// side by side, since one chain of dependent operations a warp leaves issue
// slots empty. A pixel that a record does not touch takes part with alpha
// zero, which leaves its sums and T as they are as long as the record's colour
// and depth are finite; a batch with one that is not updates pixel by pixel. Against whole 8x8 blocks visiting records
// pixel by pixel: 1M splats at 1080p 0.386 -> 0.274 ms, 6M at 4K 1.34 ->
// 1.00 ms, 100k at 512x512 0.115 -> 0.059 ms; 57 warp instructions a pair
// instead of 94. Bounds of 7 or 8 blocks an SM, without the few spilled bytes
// the compiler chooses here, are slower (0.285, 0.283).
// Each pixel runs the reference's loop unchanged over the records it is
// given, so it stops at T < 1e-4 exactly as the reference does; a warp leaves
// a batch when no cell of it has records left for pixels still blending, and
// the block stops when every pixel has.
// kTrain: also keep, per pixel, the blended colour before linearising with
// the final transmittance, and one past the last pair that contributed --
// what the backward pass re-blends from.
// kComposite: splatBlendComposite (splat_blend.slang:116-120). A disc record
// (colour.w > 0.5) that passes a pixel's cut ends its walk as an opaque hit,
// and with an under layer a pixel stops at the first pair of the tile whose
// depth is at or behind the layer's there -- whether or not that pair touches
// the pixel. Pairs are in depth-key order, not exactly depth order, so that
// first pair is found from a running maximum of the batch's depths (the first
// index where it reaches the layer's depth), not from depth order.
// Returns true when a bounded wait gave up (kErrTimeout is set): the
// barrier's phase is then unknown, so a persistent caller must stop.
// kWords: the pairs are 64-bit words with the slot (or emit index) in their
// low field; else every tile's slots alone (rows.cu).
template <bool kTrain, bool kWords, bool kComposite = false>
__device__ __forceinline__ bool blend_tile(const BlendParams& bp, uint32_t tile, uint32_t tx, uint32_t ty,
                                           const uint2* __restrict__ ranges,
                                           const unsigned long long* __restrict__ pairs,
                                           const uint32_t* __restrict__ emitSlot,
                                           const ProjRecord* __restrict__ proj, float4* __restrict__ colourOut,
                                           float* __restrict__ depthOut, float4* __restrict__ pixState,
                                           uint32_t* __restrict__ pixLast, uint32_t* __restrict__ err,
                                           BlendShared& sh, uint32_t& phase,
                                           const float4* __restrict__ underColour = nullptr,
                                           const float* __restrict__ underDepth = nullptr,
                                           CompositeShared* comp = nullptr) {
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    // Warp w holds the 8x8 block ((w & 1), (w >> 1)), its lanes 8 s.. the
    // block's cell ((s & 1), (s >> 1)).
    const uint32_t cellX = (warp & 1u) * 2u + ((lane >> 3) & 1u), cellY = (warp >> 1) * 2u + (lane >> 4);
    const uint32_t cell = cellY * 4u + cellX;
    const uint32_t px = tx * kTile + cellX * 4u + (lane & 3u);
    const uint32_t py0 = ty * kTile + cellY * 4u + ((lane >> 2) & 1u);
    const uint2 range = ranges[tile];
    const uint32_t start = range.x, end = range.y;
    const unsigned long long slotMask = (1ull << bp.slotBits) - 1ull;
    const bool depthAtThreshold = bp.depthMode != 0;   // only that mode's image reads depthAt
    const float tileX = static_cast<float>(tx * kTile), tileY = static_cast<float>(ty * kTile);
    const float2 px2 = make_float2(static_cast<float>(px) + 0.5f, static_cast<float>(px) + 0.5f);
    const float2 py2 = make_float2(static_cast<float>(py0) + 0.5f, static_cast<float>(py0 + 2u) + 0.5f);
    // The lane's two pixels: .x / [0] and, 2 rows further, .y / [1].
    float2 r = make_float2(0.0f, 0.0f), g = r, b = r, depthSum = r, T = make_float2(1.0f, 1.0f);
    float depthAt[kBlendPix];
    bool inside[kBlendPix], done[kBlendPix];
    uint32_t last[kBlendPix];
#pragma unroll
    for (uint32_t q = 0; q < kBlendPix; ++q) {
        inside[q] = px < bp.width && py0 + 2u * q < bp.height;
        done[q] = !inside[q];
        if (done[q]) (q == 0 ? T.x : T.y) = 0.0f;   // a pixel is done when its T is below 1e-4
        depthAt[q] = -1.0f;
        last[q] = start;
    }
    // Composite state: the under layer's depth here, where the layer stops
    // this pixel's walk (a pair index), and what ended the walk opaquely.
    bool underHit[kBlendPix] = {false, false}, opaqueHit[kBlendPix] = {false, false};
    float underZ[kBlendPix] = {0.0f, 0.0f}, opaqueZ[kBlendPix] = {0.0f, 0.0f};
    uint32_t stopAt[kBlendPix] = {0xFFFFFFFFu, 0xFFFFFFFFu};
    float4 opaque[kBlendPix] = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
    float zCarry = -3.4e38f;   // the largest depth of the tile's earlier batches
    if constexpr (kComposite) {
#pragma unroll
        for (uint32_t q = 0; q < kBlendPix; ++q) {
            if (underColour != nullptr && inside[q]) {
                underZ[q] = underDepth[static_cast<size_t>(py0 + 2u * q) * bp.width + px];
                underHit[q] = underZ[q] > 0.0f;
            }
        }
    }

    // The record slot of the pair at `at` + this thread's index.
    auto slot_at = [&](uint32_t at) -> uint32_t {
        if (at >= end || tid >= end - at) return 0u;
        if constexpr (!kWords) return reinterpret_cast<const uint32_t*>(pairs)[at + tid];
        uint32_t slot = static_cast<uint32_t>(pairs[at + tid] & slotMask);
        if constexpr (kTrain) {
            if (emitSlot != nullptr) slot = emitSlot[slot];   // the low field is the emit index
        }
        return slot;
    };
    auto issue = [&](uint32_t at, uint32_t slot) {
        const uint32_t cnt = min(kBatch, end - at);
        if (tid == 0) mbar_arrive_expect_tx(&sh.bar, cnt * static_cast<uint32_t>(sizeof(ProjRecord)));
        if (tid < cnt) {
            fence_proxy_async_smem();
            bulk_copy_record(&sh.rec[tid], proj + slot, &sh.bar);
        }
    };

    bool gaveUp = false;
    uint32_t nextSlot = 0;
    if (start < end) {
        issue(start, slot_at(start));
        nextSlot = slot_at(start + kBatch);
    }
    for (uint32_t at = start; at < end; at += kBatch) {
        const bool more = at + kBatch < end;
        if (!mbar_wait(&sh.bar, phase)) {
            atomicOr(err, kErrTimeout);
            gaveUp = true;
        }
        phase ^= 1u;
        const uint32_t cnt = min(kBatch, end - at);
        float myZ = -3.4e38f;
        uint32_t touched = 0;
        bool unusual = false;   // this thread's record has a colour or depth that is not finite
        if (tid < cnt) {
            const ProjRecord rec = sh.rec[tid];
            touched = cells_touched(rec, tileX, tileY);
            myZ = rec.screen.z;
            PairRecord& w = sh.walk[tid];
            w.centre = make_float4(-rec.screen.x, -rec.screen.x, -rec.screen.y, -rec.screen.y);
            w.ab = make_float4(rec.conic.x, rec.conic.x, 2.0f * rec.conic.y, 2.0f * rec.conic.y);
            w.c = make_float4(rec.conic.z, rec.conic.z, rec.screen.w,
                              kComposite && rec.colour.w > 0.5f ? -1.0f : rec.conic.w);
            w.rg = make_float4(rec.colour.x, rec.colour.x, rec.colour.y, rec.colour.y);
            w.bz = make_float4(rec.colour.z, rec.colour.z, rec.screen.z, rec.screen.z);
            unusual = !(finite(rec.colour.x) && finite(rec.colour.y) && finite(rec.colour.z) && finite(rec.screen.z));
        }
        sh.touched[(tid & ~15u) + 2u * (tid & 7u) + ((tid >> 3) & 1u)] = static_cast<uint16_t>(touched);
        if constexpr (kComposite) {
            if (underColour != nullptr) {
                // Running maximum of the depths, tile order, across batches.
                float v = myZ;
#pragma unroll
                for (uint32_t d = 1; d < 32; d <<= 1) {
                    const float o = __shfl_up_sync(0xFFFFFFFFu, v, d);
                    if (lane >= d) v = fmaxf(v, o);
                }
                if (lane == 31) comp->warpMax[warp] = v;
                __syncthreads();
                float prior = zCarry;
                for (uint32_t w = 0; w < warp; ++w) prior = fmaxf(prior, comp->warpMax[w]);
                comp->zMax[tid] = fmaxf(v, prior);
                __syncthreads();
                zCarry = comp->zMax[cnt - 1];
#pragma unroll
                for (uint32_t q = 0; q < kBlendPix; ++q) {
                    if (underHit[q] && stopAt[q] == 0xFFFFFFFFu && zCarry >= underZ[q]) {
                        uint32_t lo = 0, hi = cnt - 1;   // zMax[hi] >= underZ
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if (comp->zMax[mid] >= underZ[q]) hi = mid; else lo = mid + 1;
                        }
                        stopAt[q] = at + lo;
                    }
                    if (at >= stopAt[q]) done[q] = true;
                }
            }
        }
        const bool allFinite = __syncthreads_or(unusual ? 1 : 0) == 0;
        if (more) {
            issue(at + kBatch, nextSlot);
            nextSlot = slot_at(at + 2 * kBatch);
        }
        // The cell's list: its thread k writes the records 16 k .. 16 k + 15
        // that may touch the cell, after the earlier threads'.
        uint32_t count;
        {
            const uint32_t part = lane & (kCellThreads - 1u);
            const uint4* marks = reinterpret_cast<const uint4*>(&sh.touched[16u * part]);
            const uint4 m0 = marks[0], m1 = marks[1];
            const uint32_t word[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            uint32_t bits = 0;   // bits k and 16 + k: records k and 8 + k
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) bits |= ((word[k] >> cell) & 0x00010001u) << k;
            bits = (bits | bits >> 8) & 0xFFFFu;
            const uint32_t own = static_cast<uint32_t>(__popc(bits));
            uint32_t upTo = own;
#pragma unroll
            for (uint32_t d = 1; d < kCellThreads; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, upTo, d, kCellThreads);
                if (part >= d) upTo += o;
            }
            count = __shfl_sync(0xFFFFFFFFu, upTo, kCellThreads - 1u, kCellThreads);
            uint8_t* at = &sh.list[cell][upTo - own];
            for (; bits != 0; bits &= bits - 1u) *at++ = static_cast<uint8_t>(16u * part + __ffs(bits) - 1u);
            if (part < 3) sh.list[cell][count + part] = static_cast<uint8_t>(kBatch);
            __syncwarp();
        }
        const uint32_t listEnd = (count + 1u) & ~1u;   // from here on: the record no pixel takes
        // A record's power and alpha at the lane's pixels (splat_power's
        // operations), and which of them pass its cut.
        struct Step {
            float2 alpha;
            bool pass0, pass1;
            float4 c;
        };
        auto step = [&](uint32_t j) -> Step {
            const PairRecord& rec = sh.walk[j];
            const float4 centre = rec.centre, ab = rec.ab;
            Step st;
            st.c = rec.c;
            const float2 dx = __fadd2_rn(px2, lower2(centre)), dy = __fadd2_rn(py2, upper2(centre));
            const float2 t = __fmul2_rn(__fmul2_rn(lower2(ab), dx), dx);
            const float2 u = __ffma2_rn(__fmul2_rn(upper2(ab), dx), dy, t);
            const float2 power = __ffma2_rn(__fmul2_rn(lower2(st.c), dy), dy, u);
            st.pass0 = !(power.x > st.c.z);
            st.pass1 = !(power.y > st.c.z);
            // A power that passes lies in [0, 9] (the cut is at most 9), so the
            // exponent's argument is in range; the other pixels discard it.
            const float2 raw = lrt_scaled_exp_half2(st.c.w, power);
            st.alpha = make_float2(fminf(0.99f, raw.x), fminf(0.99f, raw.y));
            return st;
        };
        // The reference's step with that record: pixels still blending that
        // pass the cut, and whose alpha reaches 1/255, take it.
        auto blend = [&](const Step& st, uint32_t j) {
            const PairRecord& rec = sh.walk[j];
            const float4 rg = rec.rg, bz = rec.bz;
            bool take0 = !done[0] && st.pass0, take1 = !done[1] && st.pass1;
            if constexpr (kComposite) {
                take0 = take0 && at + j < stopAt[0];
                take1 = take1 && at + j < stopAt[1];
                if (st.c.w < 0.0f) {   // a disc: opaque, the walk of the pixels it covers ends here
#pragma unroll
                    for (uint32_t q = 0; q < kBlendPix; ++q) {
                        if (q == 0 ? take0 : take1) {
                            opaqueHit[q] = true;
                            opaque[q] = make_float4(rg.x, rg.z, bz.x, 1.0f);
                            opaqueZ[q] = bz.z;
                            done[q] = true;
                        }
                    }
                    take0 = take1 = false;
                }
            }
            take0 = take0 && !(st.alpha.x < 1.0f / 255.0f);
            take1 = take1 && !(st.alpha.y < 1.0f / 255.0f);
            const float2 alpha = make_float2(take0 ? st.alpha.x : 0.0f, take1 ? st.alpha.y : 0.0f);
            const float2 weight = __fmul2_rn(T, alpha);
            // rgb += weight colour, depthSum += weight z
            // (splat_blend.slang:72-74), each one multiply-add.
            if (allFinite) {
                r = __ffma2_rn(weight, lower2(rg), r);
                g = __ffma2_rn(weight, upper2(rg), g);
                b = __ffma2_rn(weight, lower2(bz), b);
                depthSum = __ffma2_rn(weight, upper2(bz), depthSum);
            } else {
                if (take0) {
                    r.x = __fmaf_rn(weight.x, rg.x, r.x);
                    g.x = __fmaf_rn(weight.x, rg.z, g.x);
                    b.x = __fmaf_rn(weight.x, bz.x, b.x);
                    depthSum.x = __fmaf_rn(weight.x, bz.z, depthSum.x);
                }
                if (take1) {
                    r.y = __fmaf_rn(weight.y, rg.y, r.y);
                    g.y = __fmaf_rn(weight.y, rg.w, g.y);
                    b.y = __fmaf_rn(weight.y, bz.y, b.y);
                    depthSum.y = __fmaf_rn(weight.y, bz.w, depthSum.y);
                }
            }
            T = __fmul2_rn(T, __ffma2_rn(alpha, make_float2(-1.0f, -1.0f), make_float2(1.0f, 1.0f)));   // T (1 - alpha)
            if (depthAtThreshold) {
                if (take0 && depthAt[0] < 0.0f && 1.0f - T.x >= bp.depthThreshold) depthAt[0] = bz.z;
                if (take1 && depthAt[1] < 0.0f && 1.0f - T.y >= bp.depthThreshold) depthAt[1] = bz.z;
            }
            if (kTrain) {
                if (take0) last[0] = at + j + 1;
                if (take1) last[1] = at + j + 1;
            }
            done[0] = (kComposite && done[0]) || T.x < 1e-4f;
            done[1] = (kComposite && done[1]) || T.y < 1e-4f;
        };
        for (uint32_t i = 0; __any_sync(0xFFFFFFFFu, i < count && !(done[0] && done[1])); i += 2) {
            const uint32_t two = *reinterpret_cast<const uint16_t*>(&sh.list[cell][min(i, listEnd)]);
            const uint32_t j0 = two & 0xFFu, j1 = two >> 8;
            const Step s0 = step(j0), s1 = step(j1);
            blend(s0, j0);
            blend(s1, j1);
        }
        if (__syncthreads_and((done[0] && done[1]) || gaveUp ? 1 : 0)) {
            if (more) {
                // Drain the batch already in flight, and count its phase: a
                // persistent block blends its next tile with the same barrier.
                if (!mbar_wait(&sh.bar, phase)) {
                    atomicOr(err, kErrTimeout);
                    gaveUp = true;
                }
                phase ^= 1u;
            }
            break;
        }
    }
#pragma unroll
    for (uint32_t q = 0; q < kBlendPix; ++q) {
        if (!inside[q]) continue;
        const size_t pix = static_cast<size_t>(py0 + 2u * q) * bp.width + px;
        if constexpr (kComposite) {
            if (!opaqueHit[q] && underHit[q]) {
                opaqueHit[q] = true;
                opaque[q] = underColour[pix];
                opaqueZ[q] = underZ[q];
            }
        }
        const float rq = q == 0 ? r.x : r.y, gq = q == 0 ? g.x : g.y, bq = q == 0 ? b.x : b.y;
        const float Tq = q == 0 ? T.x : T.y;
        const float coverage = 1.0f - Tq;
        float lr = rq, lg = gq, lb = bq;
        if (bp.linearise != 0 && coverage > 1e-6f) {
            lr = srgb_to_linear(rq / coverage) * coverage;
            lg = srgb_to_linear(gq / coverage) * coverage;
            lb = srgb_to_linear(bq / coverage) * coverage;
        }
        float4 behind = make_float4(bp.bg[0], bp.bg[1], bp.bg[2], bp.bg[3]);
        float dSum = q == 0 ? depthSum.x : depthSum.y, dAt = depthAt[q];
        if (opaqueHit[q]) {
            behind = opaque[q];
            dSum = dSum + Tq * opaqueZ[q];
            if (dAt < 0.0f) dAt = opaqueZ[q];
        }
        const float total = opaqueHit[q] ? 1.0f : coverage;
        colourOut[pix] = make_float4(lr + Tq * behind.x, lg + Tq * behind.y, lb + Tq * behind.z,
                                     coverage + Tq * behind.w);
        depthOut[pix] = bp.depthMode == 0 ? (total > 1e-6f ? dSum / total : 0.0f) : fmaxf(dAt, 0.0f);
        if (kTrain) {
            pixState[pix] = make_float4(rq, gq, bq, Tq);
            pixLast[pix] = last[q];
        }
    }
    return gaveUp;
}

// The block's batch barrier and constant record, before its first tile.
__device__ __forceinline__ void blend_init(BlendShared& sh) {
    if (threadIdx.x == 0) {
        // The record no pixel takes: every power is above its cut.
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        sh.walk[kBatch] = PairRecord{zero, zero, make_float4(0.0f, 0.0f, -1.0f, 0.0f), zero, zero};
        mbar_init(&sh.bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
}

template <bool kTrain, bool kWords, bool kChained>
__global__ void __launch_bounds__(kBlendThreads / kBlendPix)
blend_kernel(BlendParams bp, const uint2* __restrict__ ranges, const unsigned long long* __restrict__ pairs,
             const uint32_t* __restrict__ emitSlot,
             const ProjRecord* __restrict__ proj, float4* __restrict__ colourOut, float* __restrict__ depthOut,
             float4* __restrict__ pixState, uint32_t* __restrict__ pixLast, uint32_t* __restrict__ err,
             const uint32_t* __restrict__ order) {
    chained_entry<kChained>();
    __shared__ BlendShared sh;
    blend_init(sh);
    uint32_t phase = 0;
    const uint32_t tile = order != nullptr ? order[blockIdx.x] : blockIdx.x;
    blend_tile<kTrain, kWords>(bp, tile, tile % bp.tilesX, tile / bp.tilesX, ranges, pairs, emitSlot, proj, colourOut, depthOut,
                       pixState, pixLast, err, sh, phase);
}

// splatBlendComposite (splat_blend.slang:116-120): discs and an optional
// under layer (colour may be null).
template <bool kWords>
__global__ void __launch_bounds__(kBlendThreads / kBlendPix)
blend_composite_kernel(BlendParams bp, const uint2* __restrict__ ranges, const unsigned long long* __restrict__ pairs,
                       const ProjRecord* __restrict__ proj, float4* __restrict__ colourOut,
                       float* __restrict__ depthOut, const float4* __restrict__ underColour,
                       const float* __restrict__ underDepth, uint32_t* __restrict__ err,
                       const uint32_t* __restrict__ order) {
    __shared__ BlendShared sh;
    __shared__ CompositeShared comp;
    blend_init(sh);
    uint32_t phase = 0;
    const uint32_t tile = order != nullptr ? order[blockIdx.x] : blockIdx.x;
    blend_tile<false, kWords, true>(bp, tile, tile % bp.tilesX, tile / bp.tilesX, ranges, pairs, nullptr, proj, colourOut,
                            depthOut, nullptr, nullptr, err, sh, phase, underColour, underDepth, &comp);
}

// Many views in one launch: a persistent grid whose blocks take (view, tile)
// work items from a queue in order -- the views' tiles numbered one after
// another, largest views first -- and blend each as blend_kernel does
// (kTrain: as blend_kernel<true>, keeping each view's per-pixel state).
template <bool kTrain>
__global__ void __launch_bounds__(kBlendThreads / kBlendPix)
blend_batch_kernel(BlendParams bp, const ViewParams* __restrict__ views, uint32_t viewCount,
                   const uint2* __restrict__ ranges, const unsigned long long* __restrict__ pairs,
                   const ProjRecord* __restrict__ proj, uint32_t totalTiles, uint32_t* __restrict__ queue,
                   uint32_t* __restrict__ err) {
    __shared__ BlendShared sh;
    __shared__ uint32_t sItem;
    blend_init(sh);
    uint32_t phase = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sItem = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t item = sItem;
        if (item >= totalTiles) break;
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
        const bool gaveUp = blend_tile<kTrain, true>(
            vbp, item, local % v.tilesX, local / v.tilesX, ranges, pairs, nullptr, proj + v.recordBase, v.colour,
            v.depth, kTrain ? v.pixState : nullptr, kTrain ? v.pixLast : nullptr, err, sh, phase);
        // After a wait gave up the barrier's phase is unknown: take no more
        // items (the frame reports TIMEOUT and its output is undefined).
        if (__syncthreads_or(gaveUp ? 1 : 0)) return;
    }
}

}  // namespace

cudaError_t launch_ranges(const uint64_t* pairs, const uint32_t* dCount, uint32_t cap, uint32_t tileShift,
                          uint2* ranges, uint32_t tiles, cudaStream_t stream, bool rangesZeroed) {
    cudaError_t e = rangesZeroed ? cudaSuccess : launch_zero(ranges, sizeof(uint2) * tiles, stream);
    if (e != cudaSuccess || cap == 0) return e;
    const uint32_t threads = (cap + kRangeRun - 1) / kRangeRun;
    return launch_chained(ranges_kernel<true>, ranges_kernel<false>, dim3((threads + 255) / 256), dim3(256), 0, stream,
                          reinterpret_cast<const unsigned long long*>(pairs), dCount, cap, tileShift, ranges);
}

namespace {
template <bool kChained>
__global__ void publish_counters_kernel(const uint32_t* __restrict__ counters, const uint32_t* __restrict__ bands,
                                        uint32_t* hostMapped) {
    chained_entry<kChained>();
    if (threadIdx.x < 4) hostMapped[threadIdx.x] = counters[threadIdx.x];
    unsigned long long runs = 0;
    if (bands != nullptr) {
        for (uint32_t k = threadIdx.x; k < kMaxBands; k += 32) runs += bands[k];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) runs += __shfl_xor_sync(0xFFFFFFFFu, runs, d);
    }
    if (threadIdx.x == 0) hostMapped[4] = static_cast<uint32_t>(min(runs, 0xFFFFFFFFull));
    __threadfence_system();
}
}  // namespace

cudaError_t launch_publish_counters(const uint32_t* counters, const uint32_t* bands, uint32_t* hostMapped,
                                    cudaStream_t stream) {
    return launch_chained(publish_counters_kernel<true>, publish_counters_kernel<false>, dim3(1), dim3(32), 0, stream,
                          counters, bands, hostMapped);
}

namespace {
constexpr uint32_t kOrderThreads = 256;
constexpr uint32_t kOrderBuckets = 16;

__device__ __forceinline__ uint32_t order_bucket(uint32_t work) {   // floor(log2(work + 1)), at most 15
    return min(31u - static_cast<uint32_t>(__clz(work + 1u)), kOrderBuckets - 1u);
}
// A tile's work: its pair count, or (work != null) the given value.
__device__ __forceinline__ uint32_t tile_work(const uint2* __restrict__ ranges, const uint32_t* __restrict__ work,
                                              uint32_t t) {
    if (work != nullptr) return work[t];
    const uint2 r = ranges[t];
    return r.y - r.x;
}

// A block's tiles per bucket: per warp by ballots, then in shared memory.
__device__ __forceinline__ uint32_t order_block_counts(const uint2* __restrict__ ranges,
                                                       const uint32_t* __restrict__ work, uint32_t tiles,
                                                       uint32_t (&sWarp)[kOrderThreads / 32][kOrderBuckets],
                                                       uint32_t& rank) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t t = blockIdx.x * kOrderThreads + threadIdx.x;
    const uint32_t b = t < tiles ? order_bucket(tile_work(ranges, work, t)) : kOrderBuckets;
    rank = 0;
#pragma unroll
    for (uint32_t q = 0; q < kOrderBuckets; ++q) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, b == q);
        if (lane == 0) sWarp[warp][q] = static_cast<uint32_t>(__popc(m));
        if (b == q) rank = static_cast<uint32_t>(__popc(m & ((1u << lane) - 1u)));
    }
    __syncthreads();
    return b;
}

template <bool kChained>
__global__ void __launch_bounds__(kOrderThreads) tile_order_count_kernel(const uint2* __restrict__ ranges,
                                                                         const uint32_t* __restrict__ work,
                                                                         uint32_t tiles,
                                                                         uint32_t* __restrict__ blockCounts) {
    chained_entry<kChained>();
    __shared__ uint32_t sWarp[kOrderThreads / 32][kOrderBuckets];
    uint32_t rank;
    order_block_counts(ranges, work, tiles, sWarp, rank);
    if (threadIdx.x < kOrderBuckets) {
        uint32_t n = 0;
        for (uint32_t w = 0; w < kOrderThreads / 32; ++w) n += sWarp[w][threadIdx.x];
        blockCounts[blockIdx.x * kOrderBuckets + threadIdx.x] = n;
    }
}

// The tiles in the order the blend launches them: busiest first, by buckets
// of floor(log2(pairs + 1)), index order within a bucket. Blocks start in
// launch order, so the long tiles start early and the short ones fill in at
// the end. Each block reads every block's counts (from the kernel above):
// the buckets' totals give their bases, the earlier blocks' counts its own
// places in each bucket.
template <bool kChained>
__global__ void __launch_bounds__(kOrderThreads) tile_order_place_kernel(const uint2* __restrict__ ranges,
                                                                         const uint32_t* __restrict__ work,
                                                                         uint32_t tiles,
                                                                         const uint32_t* __restrict__ blockCounts,
                                                                         uint32_t* __restrict__ order) {
    chained_entry<kChained>();
    __shared__ uint32_t sWarp[kOrderThreads / 32][kOrderBuckets];
    __shared__ uint32_t sTotal[kOrderBuckets], sBefore[kOrderBuckets];
    if (threadIdx.x < kOrderBuckets) {
        sTotal[threadIdx.x] = 0;
        sBefore[threadIdx.x] = 0;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < gridDim.x * kOrderBuckets; k += kOrderThreads) {
        const uint32_t v = blockCounts[k];
        if (v == 0) continue;
        atomicAdd(&sTotal[k % kOrderBuckets], v);
        if (k / kOrderBuckets < blockIdx.x) atomicAdd(&sBefore[k % kOrderBuckets], v);
    }
    uint32_t rank;
    const uint32_t b = order_block_counts(ranges, work, tiles, sWarp, rank);   // (its barrier also ends the sums above)
    if (threadIdx.x < kOrderBuckets) {
        const uint32_t q = threadIdx.x;
        uint32_t run = sBefore[q];
        for (uint32_t h = q + 1; h < kOrderBuckets; ++h) run += sTotal[h];   // the busier buckets come first
        for (uint32_t w = 0; w < kOrderThreads / 32; ++w) {
            const uint32_t n = sWarp[w][q];
            sWarp[w][q] = run;
            run += n;
        }
    }
    __syncthreads();
    const uint32_t t = blockIdx.x * kOrderThreads + threadIdx.x;
    if (t < tiles) order[sWarp[threadIdx.x >> 5][b] + rank] = t;
}
}  // namespace

size_t tile_order_scratch_bytes(uint32_t tiles) {
    return size_t{(tiles + kOrderThreads - 1) / kOrderThreads} * kOrderBuckets * sizeof(uint32_t);
}

cudaError_t launch_tile_order(const uint2* ranges, uint32_t tiles, uint32_t* order, uint32_t* scratch,
                              cudaStream_t stream, const uint32_t* work) {
    if (tiles == 0) return cudaSuccess;
    const uint32_t blocks = (tiles + kOrderThreads - 1) / kOrderThreads;
    cudaError_t e = launch_chained(tile_order_count_kernel<true>, tile_order_count_kernel<false>, dim3(blocks), dim3(kOrderThreads), 0, stream, ranges, work,
                                   tiles, scratch);
    if (e != cudaSuccess) return e;
    return launch_chained(tile_order_place_kernel<true>, tile_order_place_kernel<false>, dim3(blocks), dim3(kOrderThreads), 0, stream, ranges, work, tiles,
                          static_cast<const uint32_t*>(scratch), order);
}

namespace {
// A training frame's tile work for the backward blend: the pairs up to the
// tile's last contributor (the largest of its pixels' saved last indices),
// a warp a tile.
template <bool kChained>
__global__ void __launch_bounds__(256) tile_backward_work_kernel(const uint2* __restrict__ ranges,
                                                                 const uint32_t* __restrict__ pixLast, uint32_t width,
                                                                 uint32_t height, uint32_t tilesX, uint32_t tiles,
                                                                 uint32_t* __restrict__ work) {
    chained_entry<kChained>();
    const uint32_t t = blockIdx.x * 8u + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31u;
    if (t >= tiles) return;
    const uint32_t x0 = (t % tilesX) * kTile, y0 = (t / tilesX) * kTile;
    const uint32_t start = ranges[t].x;
    uint32_t last = start;
#pragma unroll
    for (uint32_t k = 0; k < kTile * kTile / 32; ++k) {
        const uint32_t p = k * 32u + lane;
        const uint32_t px = x0 + (p & (kTile - 1u)), py = y0 + p / kTile;
        if (px < width && py < height) last = max(last, pixLast[static_cast<size_t>(py) * width + px]);
    }
    last = __reduce_max_sync(0xFFFFFFFFu, last);
    if (lane == 0) work[t] = last - start;
}
}  // namespace

cudaError_t launch_tile_backward_order(const uint2* ranges, const uint32_t* pixLast, uint32_t width, uint32_t height,
                                       uint32_t tilesX, uint32_t tiles, uint32_t* order, uint32_t* scratch,
                                       uint32_t* work, cudaStream_t stream) {
    if (tiles == 0) return cudaSuccess;
    cudaError_t e = launch_chained(tile_backward_work_kernel<true>, tile_backward_work_kernel<false>, dim3((tiles + 7) / 8), dim3(256), 0, stream, ranges,
                                   pixLast, width, height, tilesX, tiles, work);
    if (e != cudaSuccess) return e;
    return launch_tile_order(ranges, tiles, order, scratch, stream, work);
}

cudaError_t launch_blend(const BlendParams& bp, const uint2* ranges, const uint64_t* pairs, const ProjRecord* proj,
                         float4* colour, float* depth, uint32_t* err, cudaStream_t stream, const uint32_t* order) {
    const uint32_t tiles = bp.tilesX * bp.tilesY;
    if (tiles == 0) return cudaSuccess;
    const bool words = bp.pairShift != 0;
    return launch_chained(words ? blend_kernel<false, true, true> : blend_kernel<false, false, true>,
                          words ? blend_kernel<false, true, false> : blend_kernel<false, false, false>, dim3(tiles),
                          dim3(kBlendThreads / kBlendPix), 0, stream, bp, ranges,
                          reinterpret_cast<const unsigned long long*>(pairs), static_cast<const uint32_t*>(nullptr), proj,
                          colour, depth, static_cast<float4*>(nullptr), static_cast<uint32_t*>(nullptr), err, order);
}

cudaError_t launch_blend_composite(const BlendParams& bp, const uint2* ranges, const uint64_t* pairs,
                                  const ProjRecord* proj, float4* colour, float* depth, const float4* underColour,
                                  const float* underDepth, uint32_t* err, cudaStream_t stream, const uint32_t* order) {
    const uint32_t tiles = bp.tilesX * bp.tilesY;
    if (tiles == 0) return cudaSuccess;
    const auto kernel = bp.pairShift != 0 ? blend_composite_kernel<true> : blend_composite_kernel<false>;
    kernel<<<tiles, kBlendThreads / kBlendPix, 0, stream>>>(
        bp, ranges, reinterpret_cast<const unsigned long long*>(pairs), proj, colour, depth, underColour, underDepth,
        err, order);
    return cudaGetLastError();
}

// `blocks` counts blocks of kBlendThreads threads; the grid has kBlendPix
// times as many blocks of kBlendThreads / kBlendPix threads.
cudaError_t launch_blend_batch(const BlendParams& bp, const ViewParams* views, uint32_t viewCount, const uint2* ranges,
                               const uint64_t* pairs, const ProjRecord* proj, uint32_t totalTiles, uint32_t* queue,
                               uint32_t* err, uint32_t blocks, cudaStream_t stream) {
    if (totalTiles == 0) return cudaSuccess;
    blend_batch_kernel<false><<<blocks * kBlendPix, kBlendThreads / kBlendPix, 0, stream>>>(
        bp, views, viewCount, ranges, reinterpret_cast<const unsigned long long*>(pairs), proj, totalTiles, queue, err);
    return cudaGetLastError();
}

cudaError_t launch_blend_batch_train(const BlendParams& bp, const ViewParams* views, uint32_t viewCount,
                                     const uint2* ranges, const uint64_t* pairs, const ProjRecord* proj,
                                     uint32_t totalTiles, uint32_t* queue, uint32_t* err, uint32_t blocks,
                                     cudaStream_t stream) {
    if (totalTiles == 0) return cudaSuccess;
    blend_batch_kernel<true><<<blocks * kBlendPix, kBlendThreads / kBlendPix, 0, stream>>>(
        bp, views, viewCount, ranges, reinterpret_cast<const unsigned long long*>(pairs), proj, totalTiles, queue, err);
    return cudaGetLastError();
}

cudaError_t launch_blend_train(const BlendParams& bp, const uint2* ranges, const uint64_t* pairs,
                               const uint32_t* emitSlot, const ProjRecord* proj, float4* colour, float* depth,
                               float4* pixState, uint32_t* pixLast, uint32_t* err, cudaStream_t stream,
                               const uint32_t* order) {
    const uint32_t tiles = bp.tilesX * bp.tilesY;
    if (tiles == 0) return cudaSuccess;
    const bool words = bp.pairShift != 0;
    return launch_chained(words ? blend_kernel<true, true, true> : blend_kernel<true, false, true>,
                          words ? blend_kernel<true, true, false> : blend_kernel<true, false, false>, dim3(tiles),
                          dim3(kBlendThreads / kBlendPix), 0, stream, bp, ranges,
                          reinterpret_cast<const unsigned long long*>(pairs), emitSlot, proj, colour, depth, pixState,
                          pixLast, err, order);
}

}  // namespace lrt
