// What the projection and the pair writes share: the exact touched tiles of
// large splats a tile row at a time, the 128-bit tile masks of the others,
// the block scan and the frame look-back.
#pragma once

#include "raster_common.cuh"

#include <cuda/atomic>

namespace lrt {
namespace {

constexpr uint32_t kProjectThreads = 256;

// Splats of up to kWarpArea tiles have their tiles tested by their warp (32
// (splat, tile) pairs a step) and keep a 128-bit tile mask; larger ones are
// counted and written a tile row at a time.
constexpr uint32_t kWarpArea = 128;
constexpr uint32_t kMaskArea = kWarpArea;
static_assert(kMaskArea <= 128, "a tile mask has 128 bits");

// ---- Splats of more than kWarpArea tiles, one tile row at a time ----
//
// The tiles of a row that the exact test (tile_touched) accepts are those
// whose box of pixel centres meets the ellipse {power <= cutoff}; within the
// row's band of pixel centres, the ellipse spans one x interval [XL, XR]. In
// double precision that interval gives, with a margin m covering every
// rounding of the float test (its inputs' rounding and the power's, which
// grows with the conic's condition number), the columns that are certainly
// touched and the few around them that must be tested exactly. A row is then
// counted in O(1) plus a handful of exact tests, and its pairs are the
// certain run with the exact hits either side of it: the counts and pairs
// are the per-tile test's own, at a cost that follows the pairs, not the
// rectangle's area. Rows near the top or bottom of the ellipse, and
// ill-conditioned conics, are tested tile by tile.
struct Footprint {
    float cx, cy, a, b, c, cut;
    uint32_t x0, x1;      // the rectangle's columns
    uint32_t y0;          // its first row
    uint32_t tid;         // the splat's thread in the block
    uint32_t table;       // the splat's first row in the row table, or kNoTable
};
constexpr uint32_t kNoTable = 0xFFFFFFFFu;

struct RowPlan {
    int32_t lo, hi;           // candidate columns, inside the rectangle (none when lo > hi)
    int32_t sureLo, sureHi;   // certainly touched columns, inside [lo, hi] (none when sureLo > sureHi)
};

// The x range of tile column t's pixel centres, relative to the centre, as
// tile_touched forms it (the same float values, here exact in double).
__device__ __forceinline__ double col_lo(int32_t t, float cx) {
    return static_cast<double>(static_cast<float>(t * static_cast<int32_t>(kTile)) + 0.5f) - static_cast<double>(cx);
}
__device__ __forceinline__ double col_hi(int32_t t, uint32_t width, float cx) {
    const int32_t last = min((t + 1) * static_cast<int32_t>(kTile), static_cast<int32_t>(width)) - 1;
    return static_cast<double>(static_cast<float>(last) + 0.5f) - static_cast<double>(cx);
}

__device__ __forceinline__ RowPlan row_plan(const Footprint& fp, uint32_t ty, uint32_t width, uint32_t height) {
    RowPlan p{static_cast<int32_t>(fp.x0), static_cast<int32_t>(fp.x1), 1, 0};   // default: every column exact
    const double a = fp.a, b = fp.b, c = fp.c, k = fp.cut;
    const double det = a * c - b * b;
    if (!(a > 0.0) || !(c > 0.0) || !(k > 0.0) || !(det > 1e-6 * a * c)) return p;
    const double hx = sqrt(k * c / det), hy = sqrt(k * a / det);
    // Margin: the float test's power carries a relative error of a few
    // roundings (4 x 2^-24) times the condition number kappa, which moves
    // the boundary by at most that times half the long axis; its box
    // coordinates carry one rounding of magnitudes up to |centre| + extent.
    // Both with a factor of 8 to spare, plus a quarter pixel.
    const double lmin = 0.5 * (a + c) - sqrt(0.25 * (a - c) * (a - c) + b * b);
    if (!(lmin > 0.0)) return p;
    const double kappa = (fabs(a) + 2.0 * fabs(b) + fabs(c)) / lmin;
    const double reach = fabs(static_cast<double>(fp.cx)) + fabs(static_cast<double>(fp.cy)) + hx + hy + 64.0;
    const double m = 0.25 + 1.0e-6 * kappa * (hx + hy) + 5.0e-7 * reach;
    if (!(m < 24.0)) return p;
    const int32_t ity = static_cast<int32_t>(ty);
    const double ylo = static_cast<double>(static_cast<float>(ity * static_cast<int32_t>(kTile)) + 0.5f) -
                       static_cast<double>(fp.cy);
    const int32_t lastRow = min((ity + 1) * static_cast<int32_t>(kTile), static_cast<int32_t>(height)) - 1;
    const double yhi = static_cast<double>(static_cast<float>(lastRow) + 0.5f) - static_cast<double>(fp.cy);
    if (yhi < -hy - m || ylo > hy + m) {   // the band misses the ellipse by more than the margin
        p.lo = 1;
        p.hi = 0;
        return p;
    }
    // Near the ellipse's top or bottom the band's x extent is ill-conditioned
    // (it grows as the square root of the band's overlap): there the
    // candidates are the x extent of the band widened by m on both sides,
    // each tested exactly, and none is certain.
    const bool tangent = yhi < -hy + m || ylo > hy - m;
    const double bandLo = tangent ? fmax(ylo - m, -hy) : ylo;
    const double bandHi = tangent ? fmin(yhi + m, hy) : yhi;
    // The ellipse's x extent within the band: its leftmost and rightmost
    // points (x = -+hx, y = -b x / c) clamped into the band.
    const double yl = fmin(fmax(b * hx / c, bandLo), bandHi);
    const double yr = fmin(fmax(-b * hx / c, bandLo), bandHi);
    const double xl = (-b * yl - sqrt(fmax(k * a - det * yl * yl, 0.0))) / a;
    const double xr = (-b * yr + sqrt(fmax(k * a - det * yr * yr, 0.0))) / a;
    // First column whose hi >= v, and last whose lo <= v, within the
    // rectangle (the estimate is exact but for the clipped last column; the
    // adjustment steps are bounded and, if they do not settle, every column
    // is tested exactly).
    const int32_t x0 = static_cast<int32_t>(fp.x0), x1 = static_cast<int32_t>(fp.x1);
    bool ok = true;
    auto firstHiAtLeast = [&](double v) -> int32_t {
        const double e = ceil((v + static_cast<double>(fp.cx) - 15.5) / 16.0);
        int32_t t = static_cast<int32_t>(fmin(fmax(e, static_cast<double>(x0)), static_cast<double>(x1 + 1)));
        for (int it = 0; it < 3 && t > x0 && col_hi(t - 1, width, fp.cx) >= v; ++it) --t;
        for (int it = 0; it < 3 && t <= x1 && col_hi(t, width, fp.cx) < v; ++it) ++t;
        if ((t > x0 && col_hi(t - 1, width, fp.cx) >= v) || (t <= x1 && col_hi(t, width, fp.cx) < v)) ok = false;
        return t;
    };
    auto lastLoAtMost = [&](double v) -> int32_t {
        const double e = floor((v + static_cast<double>(fp.cx) - 0.5) / 16.0);
        int32_t t = static_cast<int32_t>(fmin(fmax(e, static_cast<double>(x0 - 1)), static_cast<double>(x1)));
        for (int it = 0; it < 3 && t < x1 && col_lo(t + 1, fp.cx) <= v; ++it) ++t;
        for (int it = 0; it < 3 && t >= x0 && col_lo(t, fp.cx) > v; ++it) --t;
        if ((t < x1 && col_lo(t + 1, fp.cx) <= v) || (t >= x0 && col_lo(t, fp.cx) > v)) ok = false;
        return t;
    };
    const int32_t lo = firstHiAtLeast(xl - m), hi = lastLoAtMost(xr + m);
    const int32_t sureLo = tangent ? 1 : firstHiAtLeast(xl + m), sureHi = tangent ? 0 : lastLoAtMost(xr - m);
    if (!ok) return p;
    p.lo = lo;
    p.hi = hi;
    p.sureLo = tangent ? 1 : max(sureLo, lo);
    p.sureHi = tangent ? 0 : min(sureHi, hi);
    return p;
}

// A row's touched tiles in column order: `visit(t)` for each exact hit and
// `run(t0, t1)` for the certain run [t0, t1].
template <class Hit, class Run>
__device__ __forceinline__ void row_walk(const Footprint& fp, uint32_t ty, uint32_t width, uint32_t height,
                                         Hit&& visit, Run&& run) {
    const RowPlan p = row_plan(fp, ty, width, height);
    const bool sure = p.sureLo <= p.sureHi;
    const int32_t leftEnd = sure ? p.sureLo - 1 : p.hi;
    for (int32_t t = p.lo; t <= leftEnd; ++t)
        if (tile_touched(width, height, fp.cx, fp.cy, fp.a, fp.b, fp.c, fp.cut, static_cast<uint32_t>(t), ty)) visit(t);
    if (!sure) return;
    run(p.sureLo, p.sureHi);
    for (int32_t t = p.sureHi + 1; t <= p.hi; ++t)
        if (tile_touched(width, height, fp.cx, fp.cy, fp.a, fp.b, fp.c, fp.cut, static_cast<uint32_t>(t), ty)) visit(t);
}

// One row: its count, first and last touched column, and whether its hits
// are one run.
struct RowCount {
    uint32_t count;
    int32_t first, last;
    bool regular;
};
__device__ __forceinline__ RowCount row_count(const Footprint& fp, uint32_t r, uint32_t width, uint32_t height) {
    RowCount rc{0, 0, -2, true};
    auto add = [&](int32_t t0, int32_t t1) {
        if (rc.count != 0 && t0 != rc.last + 1) rc.regular = false;
        if (rc.count == 0) rc.first = t0;
        rc.count += static_cast<uint32_t>(t1 - t0 + 1);
        rc.last = t1;
    };
    row_walk(fp, fp.y0 + r, width, height, [&](int32_t t) { add(t, t); }, add);
    return rc;
}
constexpr uint64_t kFlagAggregate = 1ull << 62;
constexpr uint64_t kFlagInclusive = 2ull << 62;
constexpr uint64_t kValueMask = (1ull << 62) - 1;
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* sWarp, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= d) x += o;
    }
    if (lane == 31) sWarp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kProjectThreads / 32 ? sWarp[lane] : 0;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, w, d);
            if (lane >= d) w += o;
        }
        if (lane < kProjectThreads / 32) sWarp[lane] = w;
    }
    __syncthreads();
    const uint32_t before = warp == 0 ? 0 : sWarp[warp - 1];
    *total = sWarp[kProjectThreads / 32 - 1];
    __syncthreads();
    return before + x - v;
}

// The block's first pair in the frame: warp 0 publishes the block's total
// and looks back 32 partitions at a time (lane l reads the status of
// partition q - l); the nearest inclusive prefix ends the walk and the
// aggregates up to it are summed across the warp. A partition in the window
// that has published nothing yet makes the warp read the window again
// (bounded: after kSpinLimit polls kErrTimeout is raised and the walk
// ends). The frame's last partition writes the total to counters[1], and
// raises `tooMany` where that has no room for it.
// Called by warp 0 only; lane 0's result is the block's base.
__device__ __forceinline__ unsigned long long frame_lookback(uint64_t* __restrict__ status, uint32_t g,
                                                             uint32_t lastPartition, uint32_t blockTotal,
                                                             uint32_t* __restrict__ counters,
                                                             uint32_t* __restrict__ err,
                                                             uint32_t tooMany = kErrTooManyPairs) {
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t prefix = 0;
    if (lane == 0) {
        cuda::atomic_ref<uint64_t, cuda::thread_scope_device> mine(status[g]);
        mine.store((g == 0 ? kFlagInclusive : kFlagAggregate) | blockTotal, cuda::memory_order_relaxed);
    }
    if (g > 0) {
        int64_t q = static_cast<int64_t>(g) - 1;
        uint32_t spins = 0;
        while (true) {
            const int64_t idx = q - static_cast<int64_t>(lane);
            uint64_t word = kFlagInclusive;   // before partition 0: an empty inclusive prefix
            if (idx >= 0) {
                cuda::atomic_ref<uint64_t, cuda::thread_scope_device> sref(status[idx]);
                word = sref.load(cuda::memory_order_relaxed);
            }
            const uint32_t inclusive = __ballot_sync(0xFFFFFFFFu, (word & kFlagInclusive) != 0);
            const uint32_t empty = __ballot_sync(0xFFFFFFFFu, (word & ~kValueMask) == 0);
            const uint32_t first = inclusive != 0 ? static_cast<uint32_t>(__ffs(inclusive)) - 1u : 32u;
            const uint32_t upTo = first < 32u ? (2u << first) - 1u : 0xFFFFFFFFu;   // lanes 0..first
            if ((empty & upTo) != 0) {
                if (++spins > kSpinLimit) {
                    if (lane == 0) atomicOr(err, kErrTimeout);
                    break;
                }
                __nanosleep(32);
                continue;
            }
            uint64_t v = ((upTo >> lane) & 1u) ? (word & kValueMask) : 0ull;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
            prefix += v;
            if (first < 32u) break;
            q -= 32;
        }
        if (lane == 0) {
            cuda::atomic_ref<uint64_t, cuda::thread_scope_device> mine(status[g]);
            mine.store(kFlagInclusive | (prefix + blockTotal), cuda::memory_order_relaxed);
        }
    }
    if (lane == 0 && g == lastPartition) {
        const uint64_t all = prefix + blockTotal;
        if (all > 0xFFFFFFFFull) atomicOr(err, tooMany);
        counters[1] = static_cast<uint32_t>(all);
    }
    return prefix;
}

// The position of the r-th set bit (from 0, lowest first) of a 64-bit mask
// that has more than r set bits: the half, then five halvings by population
// count.
__device__ __forceinline__ uint32_t nth_set_bit(unsigned long long m, uint32_t r) {
    uint32_t w = static_cast<uint32_t>(m);
    uint32_t base = 0;
    const uint32_t lowCount = static_cast<uint32_t>(__popc(w));
    if (r >= lowCount) {
        r -= lowCount;
        w = static_cast<uint32_t>(m >> 32);
        base = 32;
    }
#pragma unroll
    for (uint32_t width = 16; width > 0; width >>= 1) {
        const uint32_t lowBits = w & ((1u << width) - 1u);
        const uint32_t c = static_cast<uint32_t>(__popc(lowBits));
        if (r >= c) {
            r -= c;
            w >>= width;
            base += width;
        } else {
            w = lowBits;
        }
    }
    return base;
}

// The same over a 128-bit mask (lo, hi) with more than r set bits.
__device__ __forceinline__ uint32_t nth_set_bit128(unsigned long long lo, unsigned long long hi, uint32_t r) {
    const uint32_t lowCount = static_cast<uint32_t>(__popcll(lo));
    return r < lowCount ? nth_set_bit(lo, r) : 64u + nth_set_bit(hi, r - lowCount);
}

// Row and column of bit `bit` of a row-major mask of width w (w <= 128,
// bit < 128): (bit + 1/2) / w in float lies at least 1/256 away from an
// integer, far more than its rounding error, so the floor is exact.
__device__ __forceinline__ void mask_bit_tile(uint32_t bit, uint32_t w, float invW, uint32_t& dx, uint32_t& dy) {
    dy = static_cast<uint32_t>((static_cast<float>(bit) + 0.5f) * invW);
    dx = bit - dy * w;
}

// ---- Tile masks as runs ----
//
// A mask's runs: its maximal runs of touched tiles within a row of the
// rectangle. kRowStarts[w] has the bits k w (the first tile of each row) of a
// mask of width w.
struct RowStarts {
    unsigned long long lo[kMaskArea + 1], hi[kMaskArea + 1];
    constexpr RowStarts() : lo(), hi() {
        for (uint32_t w = 1; w <= kMaskArea; ++w)
            for (uint32_t k = 0; k < kMaskArea; k += w) (k < 64 ? lo[w] : hi[w]) |= 1ull << (k & 63u);
    }
};
__device__ constexpr RowStarts kRowStarts;

// The first tile of each run.
__device__ __forceinline__ ulonglong2 mask_run_starts(unsigned long long lo, unsigned long long hi, uint32_t w) {
    const unsigned long long prevLo = lo << 1, prevHi = (hi << 1) | (lo >> 63);
    return make_ulonglong2(lo & ~(prevLo & ~kRowStarts.lo[w]), hi & ~(prevHi & ~kRowStarts.hi[w]));
}
// The length of the run that starts at bit `bit`, column dx of w.
__device__ __forceinline__ uint32_t mask_run_length(unsigned long long lo, unsigned long long hi, uint32_t bit,
                                                    uint32_t dx, uint32_t w) {
    unsigned long long a = hi, b = 0;
    const uint32_t s = bit & 63u;
    if (bit < 64) {
        a = s != 0 ? (lo >> s) | (hi << (64 - s)) : lo;
        b = hi >> s;
    } else {
        a = hi >> s;
    }
    const uint32_t ones = ~a != 0 ? static_cast<uint32_t>(__ffsll(static_cast<long long>(~a))) - 1u
                          : ~b != 0 ? 63u + static_cast<uint32_t>(__ffsll(static_cast<long long>(~b))) : 128u;
    return min(ones, w - dx);
}

}  // namespace
}  // namespace lrt
