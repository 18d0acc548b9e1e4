// Stages (b) to (d) of a single frame of at most 256 x 256 tiles: from the
// depth-sorted splats to every tile's slots in depth order and its range, the
// order the reference reaches by emitting a (tile, slot) pair per touched
// tile and sorting the pairs by tile (shaders/lrt/splat/splat_emit.slang:17-50,
// modules/render/src/TileRasterizer.cpp:401-457).
//
// Sorting the pairs moves every pair through memory five times (written,
// read and written by each of two digit passes, read for the ranges) and
// ranks each against a warp's 31 others twice. But a splat's touched tiles
// are a few runs of neighbours, one a tile row. So what is sorted here are
// the runs, on their tile row only, in one digit pass; and within a tile row
// the runs, in depth order, are spread over the row's tiles by bit counting:
//
//   depth_runs_kernel   the first run of each splat in depth order (a prefix
//                       over the splats' run counts), the pair total, and
//                       each slot's first emit index (training);
//   row_runs_kernel     the runs in depth order, 2048 a block, however many
//                       splats they belong to, written to their place in the
//                       stable order by tile row (one onesweep digit pass
//                       whose keys are made, not read);
//   row_counts_kernel   2048 consecutive runs of a tile row a block: how many
//                       hold each tile, and how many before the block do, by
//                       a look-back along the row;
//   row_pairs_kernel    the same runs as a bit per (run, tile) in shared
//                       memory, each tile's set ones written out as that
//                       tile's next slots.
//
// The bits of 32 runs over a row's tiles come from two exclusive-ors a run
// (where it starts and where it has ended) and a running exclusive-or along
// the row, at a cost that does not depend on the runs' lengths. Pairs are
// written once, as 4-byte slots (and a 4-byte emit index in training frames).
//
// 6M splats at 4K (250M pairs in 31M runs): 2.03 ms (the runs 0.85, their
// spreading 1.17) and 0.13 ms more in the projection, which counts the runs,
// against 4.91 ms for writing the pairs and sorting their words (1.51 and
// 3.40). Where a splat touches a few tiles the two are alike; render_frame's
// rule says where the line lies.
#include "kernels.cuh"
#include "lookback.cuh"
#include "project_common.cuh"
#include "raster_common.cuh"

namespace lrt {
namespace {

constexpr uint32_t kRowThreads = 256;
constexpr uint32_t kRowWarps = kRowThreads / 32;
constexpr uint32_t kRunItems = 8;
constexpr uint32_t kRunTile = kRowThreads * kRunItems;   // runs a block of row_runs_kernel takes at a time
constexpr uint32_t kRunBlocks = 4;                       // its blocks an SM (64 registers a thread)
constexpr uint32_t kSpreadRuns = 2048;                   // runs of a tile row a block spreads at a time
constexpr uint32_t kSpreadWords = kSpreadRuns / 32;
constexpr uint32_t kSpreadThreads = 512;
constexpr uint32_t kSpreadWarps = kSpreadThreads / 32;
static_assert(kSpreadWords == 64, "a lane writes the runs of two words");
constexpr uint32_t kTilesPerSpread = kSpreadRuns / kRunTile;
static_assert(kTilesPerSpread * kRunTile == kSpreadRuns, "a spread holds whole tiles of runs");
// Words from one 32 runs' bits over a row's tiles to the next's: whole groups
// of eight tiles (a lane's two 16-byte accesses), and four more, which puts
// the 32 rows' words of one tile on eight banks.
__host__ __device__ constexpr uint32_t spread_stride(uint32_t tilesX) { return ((tilesX + 7u) & ~7u) + 4u; }
// row_pairs_kernel's dynamic shared memory.
constexpr size_t spread_bytes(uint32_t tilesX, bool train) {
    return (kSpreadWords * spread_stride(tilesX) + kSpreadRuns * (train ? 2u : 1u)) * sizeof(uint32_t);
}
constexpr uint32_t kOffsetItems = 8;                    // depth positions a thread of depth_runs_kernel takes
static_assert(kRowThreads == kProjectThreads && kRowThreads == kMaxBands, "a thread a tile row, the scans' block size");

// Look-back words: the value in the low half, the status above it.
constexpr unsigned long long kAggregate = 1ull << 32, kInclusive = 2ull << 32, kLookValue = 0xFFFFFFFFull;

// A run word: slot | first tile of the row << 32 | tiles << 40 (0 to 256) |
// tile row << 49.
__device__ __forceinline__ unsigned long long run_word(uint32_t slot, uint32_t x0, uint32_t count, uint32_t band) {
    return slot | (static_cast<unsigned long long>(x0) << 32) | (static_cast<unsigned long long>(count) << 40) |
           (static_cast<unsigned long long>(band) << 49);
}
__device__ __forceinline__ uint32_t run_first(unsigned long long w) { return static_cast<uint32_t>(w >> 32) & 0xFFu; }
__device__ __forceinline__ uint32_t run_count(unsigned long long w) { return static_cast<uint32_t>(w >> 40) & 0x1FFu; }
__device__ __forceinline__ uint32_t run_band(unsigned long long w) { return static_cast<uint32_t>(w >> 49) & 0xFFu; }

// The k-th run of a splat, tiles in row-major order: of a masked splat's
// mask; a larger one's k-th tile row (kept by the projection, or planned
// again); or, when its rows are not all single runs, its rectangle's k-th
// tile. Rows and tiles without a touched tile give empty runs.
__device__ __forceinline__ unsigned long long masked_run(uint32_t slot, uint32_t k, uint4 rect, ulonglong2 mask) {
    const uint32_t rw = rect.z - rect.x + 1;
    const ulonglong2 starts = mask_run_starts(mask.x, mask.y, rw);
    const uint32_t bit = nth_set_bit128(starts.x, starts.y, k);
    uint32_t dx, dy;
    mask_bit_tile(bit, rw, 1.0f / static_cast<float>(rw), dx, dy);
    return run_word(slot, rect.x + dx, mask_run_length(mask.x, mask.y, bit, dx, rw), rect.y + dy);
}
__device__ __forceinline__ unsigned long long kept_run(uint32_t slot, uint32_t k, uint4 rect, uint2 row) {
    return run_word(slot, row.y != 0 ? row.x : rect.x, row.y, rect.y + k);
}
// A large splat's run that the row table does not hold.
__device__ __noinline__ unsigned long long planned_run(const RowFrame& f, uint32_t slot, uint32_t k, uint4 rect,
                                                       bool irregular) {
    const ProjRecord rec = f.proj[slot];
    if (irregular) {
        const uint32_t rw = rect.z - rect.x + 1;
        const uint32_t tx = rect.x + k % rw, ty = rect.y + k / rw;
        const bool hit = tile_touched(f.width, f.height, rec.screen.x, rec.screen.y, rec.conic.x, rec.conic.y,
                                      rec.conic.z, rec.screen.w, tx, ty);
        return run_word(slot, tx, hit ? 1u : 0u, ty);
    }
    const Footprint fp{rec.screen.x, rec.screen.y, rec.conic.x, rec.conic.y, rec.conic.z, rec.screen.w,
                       rect.x, rect.z, rect.y, 0, kNoTable};
    const RowCount rc = row_count(fp, k, f.width, f.height);
    return kept_run(slot, k, rect, make_uint2(static_cast<uint32_t>(rc.first), rc.count));
}
// Where a splat's runs come from: its mask, the row table (row: its entry's
// place), or a plan.
enum RunKind : uint32_t { kMasked, kKept, kPlanned };
__device__ __forceinline__ RunKind run_kind(uint4 rect, ulonglong2 a, uint32_t k, uint32_t& row) {
    if ((rect.z - rect.x + 1) * (rect.w - rect.y + 1) <= kMaskArea) return kMasked;
    row = static_cast<uint32_t>(a.x >> 32);
    const bool kept = (a.x & 1ull) == 0 && row != kNoTable;
    row += k;
    return kept ? kKept : kPlanned;
}
__device__ __forceinline__ unsigned long long splat_run(const RowFrame& f, uint32_t slot, uint32_t k) {
    const uint4 rect = __ldg(f.rects + slot);
    const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2*>(f.aux) + slot);
    uint32_t row = 0;
    const RunKind kind = run_kind(rect, a, k, row);
    return kind == kMasked ? masked_run(slot, k, rect, a)
           : kind == kKept ? kept_run(slot, k, rect, __ldg(f.rowTable + row))
                           : planned_run(f, slot, k, rect, (a.x & 1ull) != 0);
}

// The scratch behind a frame's rows: zeroed before the frame ...
struct RowZeroed {
    uint64_t* pairStatus;   // look-back words of depth_runs_kernel's blocks
    uint64_t* runStatus;
    uint32_t* tickets;      // one a kernel
};
// ... and written by it.
struct RowScratch {
    unsigned long long* runLook;    // 256 words a block of row_runs_kernel (cleared by depth_runs_kernel)
    unsigned long long* tileLook;   // tilesX words a block of row_counts_kernel (cleared by row_runs_kernel)
    uint32_t* runStart;             // each depth position's first run
    uint32_t* tileSplat;            // the depth position of each kRunTile-th run's splat
    uint32_t* bandPairs;            // pairs per tile row
};

inline uint32_t offset_blocks(uint32_t slots) {
    const uint32_t perBlock = kRowThreads * kOffsetItems;
    return (slots + perBlock - 1) / perBlock;
}
inline uint32_t run_tiles(uint32_t runCap) { return runCap / kRunTile + 1; }
inline uint32_t spread_blocks(uint32_t runCap) { return runCap / kSpreadRuns + 1 + kMaxBands; }

RowZeroed row_zeroed(const RowFrame& f) {
    RowZeroed z;
    z.pairStatus = static_cast<uint64_t*>(f.zeroed);
    z.runStatus = z.pairStatus + offset_blocks(f.slots);
    z.tickets = reinterpret_cast<uint32_t*>(z.runStatus + offset_blocks(f.slots));
    return z;
}
RowScratch row_scratch(const RowFrame& f) {
    RowScratch s;
    s.runLook = static_cast<unsigned long long*>(f.scratch);
    s.tileLook = s.runLook + size_t{run_tiles(f.runCap)} * kMaxBands;
    s.runStart = reinterpret_cast<uint32_t*>(s.tileLook + size_t{spread_blocks(f.runCap)} * f.tilesX);
    s.tileSplat = s.runStart + f.slots;
    s.bandPairs = s.tileSplat + run_tiles(f.runCap);
    return s;
}

// Each depth position's first run: the exclusive prefix of the run counts
// over the depth-sorted slots, and likewise the pairs (counters[1] and, in a
// training frame, each slot's first emit index). The block also clears the
// look-back words of the row_runs_kernel blocks whose runs begin in its
// stretch and says which splat each of those begins with.
template <bool kChained>
__global__ void __launch_bounds__(kRowThreads)
depth_runs_kernel(RowFrame f, RowZeroed z, RowScratch s, uint32_t lastBlock) {
    chained_entry<kChained>();
    __shared__ uint32_t sPart;
    __shared__ uint32_t sScan[kRowWarps];
    __shared__ unsigned long long sBase[2];
    const uint32_t tid = threadIdx.x;
    if (tid == 0) sPart = atomicAdd(z.tickets, 1u);
    __syncthreads();
    if ((f.counters[2] & kErrTimeout) != 0) return;   // the depth order is not whole: no pairs
    const uint32_t part = sPart;
    const uint32_t d0 = (part * kRowThreads + tid) * kOffsetItems;
    uint32_t slot[kOffsetItems], runs[kOffsetItems], touched[kOffsetItems];
    uint32_t mine = 0, minePairs = 0;
#pragma unroll
    for (uint32_t k = 0; k < kOffsetItems; ++k) {
        const bool in = d0 + k < f.slots;
        slot[k] = in ? static_cast<uint32_t>(__ldg(f.sortedWords + d0 + k)) : 0u;
        const uint2 c = in ? __ldg(f.runCounts + slot[k]) : make_uint2(0u, 0u);
        touched[k] = c.x;
        runs[k] = c.y;
        minePairs += c.x;
        mine += c.y;
    }
    uint32_t blockRuns = 0, blockPairs = 0;
    uint32_t at = block_exclusive_scan(mine, sScan, &blockRuns);
    uint32_t atPair = block_exclusive_scan(minePairs, sScan, &blockPairs);
    // (the last block writes the totals to counters[1] and counters[4])
    if (tid < 32) {
        const unsigned long long b = frame_lookback(z.pairStatus, part, lastBlock, blockPairs, f.counters,
                                                    f.counters + 2);
        if (tid == 0) sBase[0] = b;
    } else if (tid < 64) {
        const unsigned long long b = frame_lookback(z.runStatus, part, lastBlock, blockRuns, f.counters + 3,
                                                    f.counters + 2, kErrRuns);
        if (tid == 32) sBase[1] = b;
    }
    __syncthreads();
    const uint32_t base = static_cast<uint32_t>(sBase[1]);
    if (tid == 0 && f.pairOffsets != nullptr && sBase[0] + blockPairs > f.pairCap)   // a training frame: see runs_whole
        atomicOr(f.counters + 2, kErrOverflow);
    if (sBase[1] + blockRuns > f.runCap) {   // they would not fit: the frame is drawn again
        if (tid == 0) atomicOr(f.counters + 2, kErrRuns);
        return;
    }
    at += base;
    atPair += static_cast<uint32_t>(sBase[0]);
#pragma unroll
    for (uint32_t k = 0; k < kOffsetItems; ++k) {
        if (d0 + k < f.slots) {
            s.runStart[d0 + k] = at;
            if (f.pairOffsets != nullptr) f.pairOffsets[slot[k]] = atPair;
            for (uint32_t m = (at + kRunTile - 1) / kRunTile; m * kRunTile < at + runs[k]; ++m) s.tileSplat[m] = d0 + k;
        }
        at += runs[k];
        atPair += touched[k];
    }
    for (uint32_t m = (base + kRunTile - 1) / kRunTile; m * kRunTile < base + blockRuns; ++m)
        s.runLook[static_cast<size_t>(m) * kMaxBands + tid] = 0ull;
}

// One value a thread (its tile row or tile): the sum of the earlier blocks'
// values, by look-back over their words at word[-stride], word[-2 stride],
// ... (`before` of them), and this block's inclusive sum published.
__device__ __forceinline__ uint32_t strided_lookback(unsigned long long* word, size_t stride, uint32_t before,
                                                     uint32_t count, uint32_t* err) {
    constexpr uint32_t kWords = 4;   // earlier words a step reads
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> mine(*word);
    if (before == 0) {
        mine.store(kInclusive | count, cuda::memory_order_relaxed);
        return 0;
    }
    mine.store(kAggregate | count, cuda::memory_order_relaxed);
    uint32_t prefix = 0, done = 0, spins = 0;   // words summed
    while (done < before) {
        unsigned long long words[kWords];
#pragma unroll
        for (uint32_t q = 0; q < kWords; ++q) {
            words[q] = kInclusive;   // before the first block: an inclusive zero
            if (done + q < before) {
                cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> w(*(word - (done + q + 1) * stride));
                words[q] = w.load(cuda::memory_order_relaxed);
            }
        }
        uint32_t used = 0;
        bool inclusive = false;
#pragma unroll
        for (uint32_t q = 0; q < kWords; ++q) {
            if (inclusive || used < q || (words[q] & ~kLookValue) == 0) continue;
            prefix += static_cast<uint32_t>(words[q] & kLookValue);
            used = q + 1;
            inclusive = (words[q] & kInclusive) != 0;
        }
        if (inclusive) break;
        done += used;
        if (used == 0) {
            if (++spins > kSpinLimit) {
                atomicOr(err, kErrTimeout);
                break;
            }
            __nanosleep(20);
        }
    }
    mine.store(kInclusive | static_cast<unsigned long long>(prefix + count), cuda::memory_order_relaxed);
    return prefix;
}

// Whether the frame's runs are whole: they fit, and no earlier wait gave up.
// A training frame's pairs have to fit as well: cut at the buffer's end in
// tile order, the ones left would hold emit indices up to the frame's total,
// and the backward, which may be enqueued before the counts are read, writes
// a pair's partials at its emit index. Such a frame gets no pairs (its ranges
// stay empty) and is reported as overflowed (kErrOverflow, which only a
// training frame raises before its pairs are written).
__device__ __forceinline__ bool runs_whole(const RowFrame& f, uint32_t n) {
    return n != 0 && n <= f.runCap &&
           (f.counters[2] & (kErrTimeout | kErrTooManyPairs | kErrRuns | kErrOverflow)) == 0;
}

// Bound by latency (each run gathers its splat's mask and rectangle from L2)
// and the ranking's ballots. A persistent grid takes kRunTile runs at a time
// by ticket. The splats of a tile of runs are those from tileSplat on whose
// first run lies in it; each marks its first run's place, and a running
// maximum over the places gives every run its splat.
template <bool kTrain, bool kChained>
__global__ void __launch_bounds__(kRowThreads, kRunBlocks)
row_runs_kernel(RowFrame f, RowZeroed z, RowScratch s) {
    chained_entry<kChained>();
    __shared__ unsigned long long sRun[kRunTile];
    __shared__ uint32_t sOwner[kRunTile];   // the run's splat, from the tile's first; then its emit index
    __shared__ uint32_t sWarpHist[kRowWarps][kMaxBands];
    __shared__ uint32_t sBlockStart[kMaxBands];
    __shared__ uint32_t sGlobal[kMaxBands];
    __shared__ uint32_t sScan[kRowWarps];
    __shared__ uint32_t sPart;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const uint32_t n = f.counters[4];
    if (!runs_whole(f, n)) return;
    uint32_t allRuns;
    const uint32_t bandStart = block_exclusive_scan(f.bands[tid], sScan, &allRuns);
    for (;;) {
        if (tid == 0) sPart = atomicAdd(z.tickets + 1, 1u);
        for (uint32_t i = tid; i < kRowWarps * kMaxBands; i += kRowThreads) (&sWarpHist[0][0])[i] = 0;
        for (uint32_t i = tid; i < kRunTile; i += kRowThreads) sOwner[i] = 0;
        __syncthreads();
        const uint32_t part = sPart;
        const uint32_t base = part * kRunTile;
        if (base >= n) return;
        const uint32_t here = min(kRunTile, n - base);
        // The look-back words of the stretch that as many runs fill (and, by
        // the first tile, of the rows' last, part-filled stretches).
        if (part % kTilesPerSpread == 0)
            for (uint32_t k = tid; k < f.tilesX; k += kRowThreads)
                s.tileLook[static_cast<size_t>(part / kTilesPerSpread) * f.tilesX + k] = 0ull;
        if (part == 0) {
            const size_t from = size_t{(n + kSpreadRuns - 1) / kSpreadRuns} * f.tilesX;
            const size_t last = (size_t{n} / kSpreadRuns + 1 + f.tilesY) * f.tilesX;
            for (size_t k = from + tid; k < last; k += kRowThreads) s.tileLook[k] = 0ull;
        }
        const uint32_t first = s.tileSplat[part];
        const uint32_t firstRun = s.runStart[first];   // at or before the tile's first run
        for (uint32_t d = first + 1 + tid; d < f.slots; d += kRowThreads) {
            const uint32_t at = s.runStart[d];
            if (at >= base + here) break;
            atomicMax(&sOwner[at - base], d - first);
        }
        __syncthreads();
        {   // running maximum over the places, eight a thread
            uint32_t v[kRunItems];
            uint32_t most = 0;
#pragma unroll
            for (uint32_t k = 0; k < kRunItems; ++k) {
                most = max(most, sOwner[tid * kRunItems + k]);
                v[k] = most;
            }
            uint32_t upTo = most;
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, upTo, d);
                if (lane >= d) upTo = max(upTo, o);
            }
            if (lane == 31) sScan[warp] = upTo;
            uint32_t prior = __shfl_up_sync(0xFFFFFFFFu, upTo, 1);
            if (lane == 0) prior = 0;
            __syncthreads();
            for (uint32_t w = 0; w < warp; ++w) prior = max(prior, sScan[w]);
#pragma unroll
            for (uint32_t k = 0; k < kRunItems; ++k) sOwner[tid * kRunItems + k] = max(v[k], prior);
            __syncthreads();
        }
        // The runs, two a thread at a time so that their loads overlap.
        constexpr uint32_t kAtOnce = 2;
#pragma unroll 1
        for (uint32_t p0 = tid; p0 < here; p0 += kAtOnce * kRowThreads) {
            uint32_t slot[kAtOnce], k[kAtOnce], row[kAtOnce];
            uint4 rect[kAtOnce];
            ulonglong2 a[kAtOnce];
            uint2 kept[kAtOnce];
            RunKind kind[kAtOnce];
#pragma unroll
            for (uint32_t q = 0; q < kAtOnce; ++q) {
                const uint32_t p = min(p0 + q * kRowThreads, here - 1u);
                const uint32_t d = first + sOwner[p];
                slot[q] = static_cast<uint32_t>(__ldg(f.sortedWords + d));
                k[q] = base + p - __ldg(s.runStart + d);
            }
#pragma unroll
            for (uint32_t q = 0; q < kAtOnce; ++q) {
                rect[q] = __ldg(f.rects + slot[q]);
                a[q] = __ldg(reinterpret_cast<const ulonglong2*>(f.aux) + slot[q]);
            }
#pragma unroll
            for (uint32_t q = 0; q < kAtOnce; ++q) {
                row[q] = 0;
                kind[q] = run_kind(rect[q], a[q], k[q], row[q]);
                kept[q] = kind[q] == kKept ? __ldg(f.rowTable + row[q]) : make_uint2(0u, 0u);
            }
#pragma unroll
            for (uint32_t q = 0; q < kAtOnce; ++q) {
                const unsigned long long w =
                    kind[q] == kMasked ? masked_run(slot[q], k[q], rect[q], a[q])
                    : kind[q] == kKept ? kept_run(slot[q], k[q], rect[q], kept[q])
                                       : planned_run(f, slot[q], k[q], rect[q], (a[q].x & 1ull) != 0);
                if (p0 + q * kRowThreads < here) sRun[p0 + q * kRowThreads] = w;
            }
        }
        __syncthreads();
        if constexpr (kTrain) {
            // Emit indices: the first splat's, its runs before this tile, and
            // the prefix of the tile's own pair counts.
            uint32_t before = 0;
            const uint32_t slot = static_cast<uint32_t>(f.sortedWords[first]);
            for (uint32_t k = tid; k < base - firstRun; k += kRowThreads) before += run_count(splat_run(f, slot, k));
            uint32_t sum[kRunItems], mine = 0, total, all;
#pragma unroll
            for (uint32_t k = 0; k < kRunItems; ++k) {
                sum[k] = mine;
                const uint32_t p = tid * kRunItems + k;
                mine += p < here ? run_count(sRun[p]) : 0u;
            }
            block_exclusive_scan(before, sScan, &total);
            const uint32_t at = f.pairOffsets[slot] + total + block_exclusive_scan(mine, sScan, &all);
#pragma unroll
            for (uint32_t k = 0; k < kRunItems; ++k) sOwner[tid * kRunItems + k] = at + sum[k];
            __syncthreads();
        }

        // The onesweep pass on the tile row (sort.cu's ranking): warp-striped
        // runs, past the end the last row's key, which ranks after every run.
        unsigned long long key[kRunItems];
        uint32_t emit[kRunItems], rank[kRunItems], dig[kRunItems];
#pragma unroll
        for (uint32_t j = 0; j < kRunItems; ++j) {
            const uint32_t p = warp * (kRunItems * 32) + j * 32 + lane;
            key[j] = p < here ? sRun[p] : ~0ull;
            emit[j] = kTrain ? sOwner[p] : 0u;
            dig[j] = run_band(key[j]);
        }
        const uint32_t lowerLanes = (1u << lane) - 1u;
        constexpr uint32_t kGroup = 4;
#pragma unroll
        for (uint32_t j0 = 0; j0 < kRunItems; j0 += kGroup) {
            uint32_t peers[kGroup];
#pragma unroll
            for (uint32_t q = 0; q < kGroup; ++q) peers[q] = match_digit(dig[j0 + q]);
#pragma unroll
            for (uint32_t q = 0; q < kGroup; ++q) {
                rank[j0 + q] = 0;
                if (lane == 31u - static_cast<uint32_t>(__clz(peers[q])))
                    rank[j0 + q] = atomicAdd(&sWarpHist[warp][dig[j0 + q]], static_cast<uint32_t>(__popc(peers[q])));
            }
#pragma unroll
            for (uint32_t q = 0; q < kGroup; ++q)
                rank[j0 + q] = __shfl_sync(0xFFFFFFFFu, rank[j0 + q], 31 - __clz(peers[q])) +
                               static_cast<uint32_t>(__popc(peers[q] & lowerLanes));
        }
        __syncthreads();
        uint32_t count = 0;
#pragma unroll
        for (uint32_t w = 0; w < kRowWarps; ++w) {
            const uint32_t c = sWarpHist[w][tid];
            sWarpHist[w][tid] = count;
            count += c;
        }
        uint32_t all;
        const uint32_t blockStart = block_exclusive_scan(count, sScan, &all);
        sBlockStart[tid] = blockStart;
        const uint32_t prefix = strided_lookback(s.runLook + static_cast<size_t>(part) * kMaxBands + tid, kMaxBands,
                                                 part, count, f.counters + 2);
        sGlobal[tid] = bandStart + prefix - blockStart;
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < kRunItems; ++j) {
            const uint32_t at = sBlockStart[dig[j]] + sWarpHist[warp][dig[j]] + rank[j];
            sRun[at] = key[j];
            if (kTrain) sOwner[at] = emit[j];
        }
        __syncthreads();
        for (uint32_t i = tid; i < here; i += kRowThreads) {
            const unsigned long long w = sRun[i];
            const uint32_t at = sGlobal[run_band(w)] + i;
            if (at < f.runCap) {
                f.runs[at] = w;
                if (kTrain) f.runEmit[at] = sOwner[i];
            }
        }
        __syncthreads();
    }
}

// Which runs a spreading block takes: the tile rows' runs one row after
// another, kSpreadRuns at a time within a row.
struct SpreadPlan {
    uint32_t firstBlock[kMaxBands + 1], firstRun[kMaxBands];
    uint32_t scan[kSpreadWarps];
};
template <uint32_t kThreads>
__device__ __forceinline__ void spread_plan(SpreadPlan& p, const uint32_t* __restrict__ bands) {
    const uint32_t tid = threadIdx.x;
    const uint32_t n = tid < kMaxBands ? bands[tid] : 0u;
    uint32_t blocks, runs;
    const uint32_t block = block_scan<kThreads>((n + kSpreadRuns - 1) / kSpreadRuns, p.scan, &blocks);
    const uint32_t run = block_scan<kThreads>(n, p.scan, &runs);
    if (tid < kMaxBands) {
        p.firstBlock[tid] = block;
        p.firstRun[tid] = run;
    }
    if (tid == 0) p.firstBlock[kMaxBands] = blocks;
    __syncthreads();
}
struct Stretch {
    uint32_t band, index, first, count, last;   // index: within the tile row; last: the row's last block
};
__device__ __forceinline__ Stretch spread_stretch(const SpreadPlan& p, const uint32_t* __restrict__ bands,
                                                  uint32_t block) {
    uint32_t lo = 0, hi = kMaxBands;   // the last tile row whose first block is at or before this one
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (p.firstBlock[mid] <= block) lo = mid; else hi = mid;
    }
    Stretch t;
    t.band = lo;
    t.index = block - p.firstBlock[lo];
    t.first = p.firstRun[lo] + t.index * kSpreadRuns;
    t.count = min(kSpreadRuns, bands[lo] - t.index * kSpreadRuns);
    t.last = p.firstBlock[lo + 1] - 1u;
    return t;
}

// A tile's runs in a stretch are those that start at or before it less those
// that have ended: two counts a run and a prefix over the tiles.
template <bool kChained>
__global__ void __launch_bounds__(kRowThreads)
row_counts_kernel(RowFrame f, RowZeroed z, RowScratch s) {
    chained_entry<kChained>();
    __shared__ SpreadPlan plan;
    __shared__ uint32_t sSteps[kMaxBands];
    __shared__ uint32_t sPart;
    const uint32_t tid = threadIdx.x;
    const uint32_t n = f.counters[4];
    if (!runs_whole(f, n)) return;
    spread_plan<kRowThreads>(plan, f.bands);
    for (;;) {
        if (tid == 0) sPart = atomicAdd(z.tickets + 2, 1u);
        sSteps[tid] = 0;
        __syncthreads();
        const uint32_t part = sPart;
        if (part >= plan.firstBlock[kMaxBands]) return;
        const Stretch t = spread_stretch(plan, f.bands, part);
#pragma unroll
        for (uint32_t q = 0; q < kSpreadRuns / kRowThreads; ++q) {
            const uint32_t p = q * kRowThreads + tid;
            if (p < t.count) {
                const unsigned long long w = __ldg(reinterpret_cast<const unsigned long long*>(f.runs) + t.first + p);
                const uint32_t x0 = run_first(w), to = x0 + run_count(w);
                if (to != x0) {
                    atomicAdd(&sSteps[x0], 1u);
                    if (to < kMaxBands) atomicSub(&sSteps[to], 1u);
                }
            }
        }
        __syncthreads();
        uint32_t all;
        const uint32_t step = sSteps[tid];
        const uint32_t count = block_exclusive_scan(step, plan.scan, &all) + step;
        uint32_t upTo = 0;
        if (tid < f.tilesX)
            upTo = count + strided_lookback(s.tileLook + static_cast<size_t>(part) * f.tilesX + tid, f.tilesX, t.index,
                                            count, f.counters + 2);
        if (part == t.last) {
            uint32_t pairs;
            block_exclusive_scan(upTo, plan.scan, &pairs);
            if (tid == 0) s.bandPairs[t.band] = pairs;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ uint32_t spread_row(uint32_t w) { return 32u * (w & 1u) + (w >> 1); }

// Bound by instruction issue: a step of the writing loop stores one pair a
// lane that has one left, and the tile's lanes hold one to a few each.
template <bool kTrain, bool kChained>
__global__ void __launch_bounds__(kSpreadThreads)
row_pairs_kernel(RowFrame f, RowZeroed z, RowScratch s) {
    chained_entry<kChained>();
    extern __shared__ __align__(16) unsigned char spreadSmem[];
    // Bit b of row 32 (w & 1) + w / 2, word c: run 32 w + b holds tile c (so
    // that a warp's 32 lanes read the rows of 64 consecutive runs each).
    uint32_t* const sBits = reinterpret_cast<uint32_t*>(spreadSmem);
    const uint32_t stride = spread_stride(f.tilesX);
    uint32_t* const sSlot = sBits + kSpreadWords * stride;   // the runs' slots
    uint32_t* const sEmit = sSlot + kSpreadRuns;   // training frames: their first emit index less their first tile
    __shared__ SpreadPlan plan;
    __shared__ uint32_t sPart;
    __shared__ uint32_t sStart[kMaxBands], sBandStart[kMaxBands + 1];
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const uint32_t n = f.counters[4];
    if (!runs_whole(f, n)) return;
    spread_plan<kSpreadThreads>(plan, f.bands);
    uint32_t all;
    {
        const bool has = tid < kMaxBands && f.bands[tid] != 0;
        const uint32_t start = block_scan<kSpreadThreads>(has ? s.bandPairs[tid] : 0u, plan.scan, &all);
        if (tid < kMaxBands) sBandStart[tid] = start;
        if (tid == 0) sBandStart[kMaxBands] = all;
    }
    for (;;) {
        if (tid == 0) sPart = atomicAdd(z.tickets + 3, 1u);
        __syncthreads();
        const uint32_t part = sPart;
        if (part >= plan.firstBlock[kMaxBands]) return;
        const Stretch t = spread_stretch(plan, f.bands, part);
        // The bits: where a run starts and where it has ended toggle its bit,
        // and a running exclusive-or along the row fills in between.
        const uint32_t words = (t.count + 31u) / 32u;
        for (uint32_t w = warp; w < kSpreadWords; w += kSpreadWarps) {   // words past the runs: zero
            uint4* row = reinterpret_cast<uint4*>(sBits + spread_row(w) * stride);
            for (uint32_t k = lane; k < stride / 4; k += 32) row[k] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < kSpreadRuns / kSpreadThreads; ++q) {
            const uint32_t p = q * kSpreadThreads + tid;
            if (p < t.count) {
                const unsigned long long w = __ldg(reinterpret_cast<const unsigned long long*>(f.runs) + t.first + p);
                const uint32_t x0 = run_first(w), to = x0 + run_count(w);
                uint32_t* row = sBits + spread_row(p >> 5) * stride;
                if (to != x0) {
                    atomicXor(row + x0, 1u << lane);   // p and the lane agree in their low five bits
                    if (to < f.tilesX) atomicXor(row + to, 1u << lane);
                }
                sSlot[p] = static_cast<uint32_t>(w);
                if constexpr (kTrain) sEmit[p] = __ldg(f.runEmit + t.first + p) - x0;
            }
        }
        // Where each tile's pairs begin, and this stretch's among them.
        uint32_t before = 0, total = 0;
        if (tid < f.tilesX) {
            if (t.index != 0)
                before = static_cast<uint32_t>(s.tileLook[static_cast<size_t>(part - 1) * f.tilesX + tid] & kLookValue);
            total = static_cast<uint32_t>(s.tileLook[static_cast<size_t>(t.last) * f.tilesX + tid] & kLookValue);
        }
        const uint32_t start = sBandStart[t.band] + block_scan<kSpreadThreads>(total, plan.scan, &all);
        if (tid < f.tilesX) {
            sStart[tid] = start + before;
            if (t.index == 0 && total != 0)
                f.ranges[t.band * f.tilesX + tid] = make_uint2(min(start, f.pairCap), min(start + total, f.pairCap));
        }
        for (uint32_t w = warp; w < words; w += kSpreadWarps) {   // (the scan's barriers ended the toggles)
            uint4* row = reinterpret_cast<uint4*>(sBits + spread_row(w) * stride + 8 * lane);
            const bool in = 8 * lane < f.tilesX;
            uint4 a = make_uint4(0, 0, 0, 0), b = a;
            if (in) {
                a = row[0];
                b = row[1];
            }
            a.y ^= a.x;
            a.z ^= a.y;
            a.w ^= a.z;
            b.x ^= a.w;
            b.y ^= b.x;
            b.z ^= b.y;
            b.w ^= b.z;
            uint32_t upTo = b.w;
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, upTo, d);
                if (lane >= d) upTo ^= o;
            }
            const uint32_t prior = upTo ^ b.w;
            if (in) {
                row[0] = make_uint4(a.x ^ prior, a.y ^ prior, a.z ^ prior, a.w ^ prior);
                row[1] = make_uint4(b.x ^ prior, b.y ^ prior, b.z ^ prior, b.w ^ prior);
            }
        }
        __syncthreads();
        // Whether the whole tile row's pairs lie inside the buffer.
        const uint32_t rowEnd = sBandStart[t.band + 1u];
        const bool fits = rowEnd <= f.pairCap && rowEnd >= sBandStart[t.band];
        // A warp a tile: lane l writes the runs 64 l .. 64 l + 63 that hold
        // it, after the lower lanes' (a step's writes lie within the tile's
        // few hundred bytes of this stretch).
#pragma unroll 1
        for (uint32_t c = warp; c < f.tilesX; c += kSpreadWarps) {
            const uint32_t* bits = sBits + lane * stride + c;
            uint32_t word = __brev(bits[0]), next = __brev(bits[32u * stride]);   // the first run in the top bit
            const uint32_t own = static_cast<uint32_t>(__popc(word) + __popc(next));
            uint32_t upTo = own;
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, upTo, d);
                if (lane >= d) upTo += o;
            }
            uint32_t at = sStart[c] + upTo - own;
            uint32_t p0 = 64u * lane;
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                if (fits) {
                    while (word != 0) {
                        const uint32_t b = static_cast<uint32_t>(__clz(word));
                        word ^= 0x80000000u >> b;
                        f.pairSlots[at] = sSlot[p0 + b];
                        if constexpr (kTrain) f.pairEmit[at] = sEmit[p0 + b] + c;
                        ++at;
                    }
                } else {
                    for (; word != 0; ++at) {
                        const uint32_t b = static_cast<uint32_t>(__clz(word));
                        word ^= 0x80000000u >> b;
                        if (at < f.pairCap) {
                            f.pairSlots[at] = sSlot[p0 + b];
                            if constexpr (kTrain) f.pairEmit[at] = sEmit[p0 + b] + c;
                        }
                    }
                }
                word = next;
                p0 += 32u;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) pair_words_kernel(const uint2* __restrict__ ranges,
                                                         const uint32_t* __restrict__ low, uint32_t tiles,
                                                         uint32_t pairs, unsigned long long* __restrict__ words) {
    const uint32_t t = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (t >= tiles) return;
    const uint2 r = ranges[t];
    for (uint32_t k = r.x + (threadIdx.x & 31u); k < min(r.y, pairs); k += 32)
        words[k] = (static_cast<unsigned long long>(t) << 32) | low[k];
}

}  // namespace

size_t row_zeroed_bytes(uint32_t slots) { return size_t{offset_blocks(slots)} * 16 + 16; }
size_t row_scratch_bytes(uint32_t slots, uint32_t runCap, uint32_t tilesX) {
    return size_t{run_tiles(runCap)} * (kMaxBands * 8 + 4) + size_t{spread_blocks(runCap)} * tilesX * 8 +
           size_t{slots} * 4 + kMaxBands * 4;
}

cudaError_t launch_row_runs(const RowFrame& f, cudaStream_t stream) {
    if (f.slots == 0) return cudaSuccess;
    const RowZeroed z = row_zeroed(f);
    const RowScratch s = row_scratch(f);
    const uint32_t blocks = offset_blocks(f.slots);
    cudaError_t e = launch_chained(depth_runs_kernel<true>, depth_runs_kernel<false>, dim3(blocks), dim3(kRowThreads),
                                   0, stream, f, z, s, blocks - 1);
    if (e != cudaSuccess) return e;
    const dim3 grid(std::min(run_tiles(f.runCap), kSms * kRunBlocks));
    return f.runEmit != nullptr
               ? launch_chained(row_runs_kernel<true, true>, row_runs_kernel<true, false>, grid, dim3(kRowThreads), 0,
                                stream, f, z, s)
               : launch_chained(row_runs_kernel<false, true>, row_runs_kernel<false, false>, grid, dim3(kRowThreads),
                                0, stream, f, z, s);
}

cudaError_t launch_row_pairs(const RowFrame& f, cudaStream_t stream) {
    if (f.slots == 0) return cudaSuccess;
    const RowZeroed z = row_zeroed(f);
    const RowScratch s = row_scratch(f);
    const uint32_t most = f.runCap / kSpreadRuns + 1 + f.tilesY;
    cudaError_t e = launch_chained(row_counts_kernel<true>, row_counts_kernel<false>, dim3(std::min(most, kSms * 8u)),
                                   dim3(kRowThreads), 0, stream, f, z, s);
    if (e != cudaSuccess) return e;
    const size_t smem = spread_bytes(f.tilesX, f.pairEmit != nullptr);
    // As many blocks as the SMs hold at once: the dynamic shared memory, the
    // kernel's own and 1 KB a block, of 228 KB; 2048 threads.
    constexpr size_t kOwn = sizeof(SpreadPlan) + (2 * kMaxBands + 2) * sizeof(uint32_t) + 1024;
    const uint32_t perSm = static_cast<uint32_t>(std::min<size_t>(2048 / kSpreadThreads, (228u << 10) / (smem + kOwn)));
    const dim3 grid(std::min(most, kSms * perSm));
    auto launch = [&](auto chained, auto plain) -> cudaError_t {
        // The limit belongs to the process, and a thread with another handle
        // may be between these lines with a frame of another width: always
        // the widest frame's.
        for (auto kernel : {chained, plain}) {
            const cudaError_t a = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       static_cast<int>(spread_bytes(kMaxBands, true)));
            if (a != cudaSuccess) return a;
        }
        return launch_chained(chained, plain, grid, dim3(kSpreadThreads), smem, stream, f, z, s);
    };
    return f.pairEmit != nullptr
               ? launch(row_pairs_kernel<true, true>, row_pairs_kernel<true, false>)
               : launch(row_pairs_kernel<false, true>, row_pairs_kernel<false, false>);
}

cudaError_t launch_pair_words(const uint2* ranges, const uint32_t* low, uint32_t tiles, uint32_t pairs,
                              uint64_t* words, cudaStream_t stream) {
    if (tiles == 0 || pairs == 0) return cudaSuccess;
    pair_words_kernel<<<(tiles + 7) / 8, 256, 0, stream>>>(ranges, low, tiles, pairs,
                                                          reinterpret_cast<unsigned long long*>(words));
    return cudaGetLastError();
}

}  // namespace lrt
