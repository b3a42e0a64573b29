// What an additive mask leaves to do, found out once per call ahead of the attention kernel (fa_fwd_pipelined with
// kMaskPlanned).  The mask is shared by the heads, so one pass over it saves every head's pass over
//   - key tiles (128 keys) that the mask takes away from all 256 query rows of a work item: half of a causal mask,
//     the padding of a batch.  They are left out: P would be 0 there, so neither l nor O changes;
//   - the mask tiles that are zero throughout (nothing is added) or -inf throughout (no tile is fetched), and those whose
//     every row is a run of zeros between -inf, of which only the runs' ends are passed on.
// A mask whose rows TMA cannot fetch (row starts on no 16-byte boundary) is copied on the way, the tiles that are
// neither, into rows that it can.
//
// Leaving a key tile out is only the same as adding -inf while its K and V are finite: 0 * inf and inf - inf are
// NaN.  So the K and V rows of every key tile that might be left out for some query tile are looked through as well (by
// the plan, or by items of the planned kernel, see plan_looks_through), and a tile with an infinity or a NaN in it is not
// left out.  (Q need not be looked at: a row of Q with an infinity
// or a NaN has no finite score, so its result is NaN whatever is left out.)
#pragma once

#include "fa_kernels.cuh"

namespace fa {

struct PlanArgs {
    const __half* mask;    // [B, L, L]
    const __half* k;       // [B, L, F]
    const __half* v;
    __half* copy;          // [B, L, copy_pitch] or nullptr: rows that start on 16-byte boundaries
    uint8_t* cls;          // [B][n][n] (query tile, key tile): kTileNeg, kTileZero, kTileMixed or kTileRows
    uint16_t* runs;        // [B][n][n][128] for a kTileRows tile: first zero | key behind the last << 8; or nullptr
    uint32_t* head;        // {1 = the planned kernel runs, 0 = the one behind it}, see kPlanInputs
    uint32_t* ticket;      // CTAs that are through; zero between launches
    uint32_t* bad;         // [B][n]: `stamp` if the key tile's K or V is not finite throughout
    uint32_t* order;       // [B * q_pairs]: (query pair of a batch entry) | key steps << kPlanLenShift, longest first
    uint16_t* list;        // [B * q_pairs][n]: key steps, see kStepShift0
    uint32_t B, L, F, n, q_pairs, copy_pitch;
    uint32_t stamp;        // of this call alone (a leftover that equals it costs a step, no more)
};
constexpr uint8_t kTileNeg = 0, kTileZero = 1, kTileMixed = 2, kTileRows = 3;
constexpr uint32_t kPlanThreads = 256;
// CTAs per SM, 32 KB of loads in flight each; the instance that copies keeps a tile in registers, which fewer leave room for
// (B=4 R=12 L=1021 H=64, the whole call: 40.5 us with four, 39.2 with three, 40.8 with two).
constexpr uint32_t kPlanCtasPerSm = 4, kPlanCopyCtasPerSm = 3;
constexpr uint32_t kPlanCols = 128;         // columns of K or V that are looked through at a time
constexpr uint32_t kPlanMaxTiles = 256;     // key tiles per sequence,
constexpr uint32_t kPlanMaxGroups = 1024;   // and pairs of query tiles of all batch entries that the lists are built for

// A row whose zeros follow one another and whose other keys are -inf is kept as its run: first zero | key behind the last
// << 8 (0: no zero).
constexpr uint32_t kWholeRun = kTile << 8;

// A tile is brought into shared memory with asynchronous copies and looked at there, in loops: a CTA of this kernel meets
// all of its code for the first time, and its length counts.  (Rows in registers and everything written out over them were
// 118 KB of code; a tile on the diagonal of B=4 R=12 L=1021 H=64 took 15 us.)
// Measured, the call: B=4 R=32 L=2048 H=128 causal 243 us with mask tiles on the diagonal and K and V looked through here,
// 209 with runs and K and V looked through by the items; this kernel alone 38 and 23.
// Words of a staged row.  Rows on 16-byte boundaries: 64.  Others in whole aligned words, where word j of a row that starts
// in the middle of one holds its keys 2 j - 1 and 2 j: 65 (and one so that rows lie an even number of banks apart).
constexpr uint32_t kPlanRowWords = 66;

// A warp's 16 rows of a 128 x 128 tile of the mask.
struct PlanRows {
    uint64_t first, pitch;   // the first of them, and from row to row, in bytes
    uint32_t b, row0, key0, rows, keys;
    bool words;   // whole words are only copied where all of them lie inside the mask: not in its first and last rows if it
                  // begins or ends in the middle of one, which are put into place value by value
    // how far into its first word a row starts
    __device__ __forceinline__ uint32_t shift(uint32_t r) const { return words ? static_cast<uint32_t>((first + r * pitch) >> 1) & 1u : 0u; }
};
__device__ __forceinline__ PlanRows plan_rows(const PlanArgs& a, uint32_t tile) {
    const uint32_t kt = tile % a.n, qt = (tile / a.n) % a.n;
    PlanRows t;
    t.b = tile / (a.n * a.n);
    t.row0 = qt * kTile + (threadIdx.x >> 5) * 16u, t.key0 = kt * kTile;
    t.rows = t.row0 < a.L ? min(16u, a.L - t.row0) : 0u;
    t.keys = min(kTile + 0u, a.L - t.key0);
    t.first = reinterpret_cast<uint64_t>(a.mask) + 2ull * ((static_cast<uint64_t>(t.b) * a.L + t.row0) * a.L + t.key0);
    t.pitch = 2ull * a.L;
    const uint64_t mask0 = reinterpret_cast<uint64_t>(a.mask);
    t.words = (t.first & ~3ull) >= mask0 &&
              ((t.first + (t.rows ? t.rows - 1u : 0u) * t.pitch + 2u * t.keys + 3u) & ~3ull) <= mask0 + 2ull * a.B * a.L * a.L;
    return t;
}

// Asks for a tile.  `staged`: this warp's rows.
template <bool kCopy>
__device__ __forceinline__ void plan_fetch_tile(const PlanRows& t, uint32_t* staged) {
    const uint32_t lane = threadIdx.x & 31u;
    if constexpr (!kCopy) {   // two rows a copy, eight keys a lane (L is a multiple of 8)
        const uint32_t piece = lane & 15u;
        const bool in = piece * 8u < t.keys;
#pragma unroll 2
        for (uint32_t r = lane >> 4; r < t.rows; r += 2u)
            cp_async_16_zero(smem_u32(staged + r * 64u + piece * 4u), reinterpret_cast<const void*>(t.first + r * t.pitch + (in ? piece * 16u : 0u)), in);
    } else if (t.words) {
        // Up to the word with the row's last key; what lies behind it in shared memory is not looked at.  (With the last word
        // copied again into every place behind it, 64 copies a row from one address where the last tile has few keys, the
        // plan of B=8 R=12 L=389 H=64 took 8 us longer: the dense call 46 us instead of 38, causal 32 instead of 26.)
#pragma unroll 2
        for (uint32_t r = 0; r < t.rows; ++r) {
            const uint64_t row = (t.first + r * t.pitch) & ~3ull;
            const uint32_t last = (t.keys + t.shift(r) - 1u) >> 1, at = smem_u32(staged + r * kPlanRowWords + lane);
            if (lane <= last) cp_async_4(at, row + 4u * lane);
            if (32u + lane <= last) cp_async_4(at + 128u, row + 4u * (32u + lane));
            if (lane == 0 && last == 64u) cp_async_4(at + 256u, row + 256u);
        }
    } else {
#pragma unroll 4
        for (uint32_t r = 0; r < t.rows; ++r) {
            const uint16_t* row = reinterpret_cast<const uint16_t*>(t.first + r * t.pitch);
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t key = h * 64u + lane * 2u;
                const uint32_t lo = key < t.keys ? ld_settled(row + key) : 0u, hi = key + 1u < t.keys ? ld_settled(row + key + 1u) : 0u;
                staged[r * kPlanRowWords + h * 32u + lane] = lo | (hi << 16);
            }
        }
    }
}

// What the tile is: its class, its rows as runs or its copy.
template <bool kCopy>
__device__ __forceinline__ void plan_look_at_tile(const PlanArgs& a, const PlanRows& t, uint32_t tile, const uint32_t* staged) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, rows = t.rows, keys = t.keys;
    cp_async_wait_all();
    __syncwarp();
    // keys 2 j and 2 j + 1 of row r (a key beyond the end: anything)
    auto two_keys = [&](uint32_t r, uint32_t j) {
        if constexpr (!kCopy) return staged[r * 64u + j];
        const uint32_t* at = staged + r * kPlanRowWords + j;
        return __funnelshift_r(at[0], at[1], t.shift(r) * 16u);
    };
    auto valid_of = [&](uint32_t key) { return (key < keys ? 0xFFFFu : 0u) | (key + 1u < keys ? 0xFFFF0000u : 0u); };   // key, key + 1
    const uint32_t valid0 = valid_of(2u * lane), valid1 = valid_of(64u + 2u * lane);
    uint32_t not_neg = 0, not_zero = 0;
#pragma unroll 4
    for (uint32_t r = 0; r < rows; ++r) {
        const uint32_t v0 = two_keys(r, lane), v1 = two_keys(r, 32u + lane);
        not_neg |= ((v0 ^ 0xFC00FC00u) & valid0) | ((v1 ^ 0xFC00FC00u) & valid1);
        not_zero |= (v0 & 0x7FFF7FFFu & valid0) | (v1 & 0x7FFF7FFFu & valid1);
    }
    const bool any_not_neg = __syncthreads_or(not_neg != 0u), any_not_zero = __syncthreads_or(not_zero != 0u);
    if (!any_not_neg || !any_not_zero) {
        if (tid == 0) a.cls[tile] = any_not_neg ? kTileZero : kTileNeg;
        return;
    }
    // Neither: rows that are runs of zeros between -inf (a causal mask's diagonal, the end of a padded sequence, a window)
    // are passed on as the ends of their runs, 256 bytes instead of 32 KB and nothing to be fetched ahead of a step.
    bool in_runs = a.runs != nullptr;
    if (in_runs) {
        // a row and half of its keys per lane (a row per warp with votes is five times the instructions)
        const uint32_t r = lane >> 1, half = (lane & 1u) * 64u;
        uint32_t from = kTile, behind = 0, count = 0;
        const uint32_t* at = staged + r * (kCopy ? kPlanRowWords : 64u) + half / 2u;
        const uint32_t sh = kCopy ? t.shift(r) * 16u : 0u;
        uint32_t w = at[0];
        // A tile of other values (a bias) shows one among the first of each half row nearly always, and is not gone through.
        // (Dense masks, us with and without the walk: B=4 R=16 L=1501 H=32 108 / 101, B=8 R=12 L=511 H=64 38.6 / 35.4.)
        const uint32_t first = (w >> sh) & 0xFFFFu;
        bool fits = __all_sync(0xffffffffu, r >= rows || half >= keys || (first & 0x7FFFu) == 0u || first == 0xFC00u);
        if (fits && r < rows) {
#pragma unroll 4
            for (uint32_t j = 0; j < 32u; ++j) {
                uint32_t v = w;
                if constexpr (kCopy) {
                    w = at[j + 1u];
                    v = __funnelshift_r(v, w, sh);
                } else {
                    w = at[min(j + 1u, 31u)];
                }
                const uint32_t key = half + 2u * j, valid = valid_of(key);
                const __half2 h = *reinterpret_cast<const __half2*>(&v);
                const uint32_t zero = __heq2_mask(h, __float2half2_rn(0.f)) & valid, neg = __heq2_mask(h, __float2half2_rn(-INFINITY));
                fits &= ((zero | neg | ~valid) == 0xFFFFFFFFu);
                if (zero) {
                    from = min(from, key + ((zero & 1u) ? 0u : 1u));
                    behind = key + ((zero >> 16) ? 2u : 1u);
                    count += (zero & 1u) + (zero >> 31);
                }
            }
        }
        from = min(from, __shfl_xor_sync(0xffffffffu, from, 1));
        behind = max(behind, __shfl_xor_sync(0xffffffffu, behind, 1));
        count += __shfl_xor_sync(0xffffffffu, count, 1);
        fits &= count == 0u || count == behind - from;
        in_runs = __syncthreads_and(fits);
        if (in_runs && half == 0u)
            a.runs[static_cast<size_t>(tile) * kTile + warp * 16u + r] = static_cast<uint16_t>(r >= rows ? kWholeRun : (count == 0u ? 0u : from | (behind << 8)));
    }
    if (tid == 0) a.cls[tile] = in_runs ? kTileRows : kTileMixed;
    if constexpr (kCopy) {
        if (in_runs) return;
        uint16_t* dst = reinterpret_cast<uint16_t*>(a.copy) + (static_cast<size_t>(t.b) * a.L + t.row0) * a.copy_pitch + t.key0;
#pragma unroll 2
        for (uint32_t r = 0; r < rows; ++r) {
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t v = two_keys(r, h * 32u + lane), at = h * 64u + lane * 2u;
                if (at < keys)   // (the pitch is even: the second key has a place)
                    *reinterpret_cast<uint32_t*>(dst + static_cast<size_t>(r) * a.copy_pitch + at) = v;
            }
        }
    }
}

// Does the plan itself look through K and V of key tile kt of batch entry b?  Only tiles that begin with -inf can be -inf
// throughout.  Where a kernel without a plan stands behind the planned one, it is done here for key tiles that may be left
// out by every item; of the others an item that works on them (plan_checker) looks them through while it multiplies: 134 MB
// of K and V at B=4 R=32 L=2048 H=128 are 25 us for a kernel of their own.
template <bool kCopy>
__device__ __forceinline__ bool plan_looks_through(const PlanArgs& a, uint32_t b, uint32_t kt) {
    bool any = false, all = true;
    for (uint32_t qt = threadIdx.x; qt < a.n; qt += kPlanThreads) {
        const bool neg = ld_settled(reinterpret_cast<const uint16_t*>(a.mask) + (static_cast<size_t>(b) * a.L + qt * kTile) * a.L + kt * kTile) == 0xFC00u;
        any |= neg, all &= neg;
    }
    return kCopy ? __syncthreads_or(any) : __syncthreads_and(all);
}

// 128 rows x up to kPlanCols columns of K or V: is every value finite?
__device__ __forceinline__ void plan_finite(const PlanArgs& a, const __half* x, uint32_t b, uint32_t kt, uint32_t c0) {
    const uint32_t tid = threadIdx.x;
    const uint32_t c = c0 + (tid & 15u) * 8u, rows = min(kTile + 0u, a.L - kt * kTile);   // F is a multiple of 16
    const __half* src = x + (static_cast<size_t>(b) * a.L + kt * kTile) * a.F + c;
    uint32_t bits = 0;
    uint4 w[8];
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
        const uint32_t r = u * 16u + (tid >> 4);
        w[u] = r < rows && c < a.F ? ld_settled(reinterpret_cast<const uint4*>(src + static_cast<size_t>(r) * a.F)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) bits |= nonfinite_bits(w[u]);
    if (bits & 0x80008000u) a.bad[b * a.n + kt] = a.stamp;
}

// The tiles of the mask, of all batch entries, that are looked at to find out whether enough of it is -inf: all of them, or
// one per thread.  Those are points of Roberts' sequence in three dimensions (multiples of the powers of the root of
// x^4 = x + 1, without their whole parts), one coordinate each for batch entry, query tile and key tile, so that they are
// spread over each of them, and over each pair, alike whatever B and n are.  (Every so-many-th tile in the order of memory
// has one key tile only where B n is a multiple of 256, and causal masks of such calls looked as if nothing were left out:
// B=16 R=8 L=2048 H=64 235 us instead of 172.)  For causal, padding and window masks and every B and n that are planned
// the share of tiles that begin with -inf is met within 0.06.
struct PlanSample { uint32_t b, qt, kt; };   // batch entry, query tile, key tile
__host__ __device__ inline uint32_t plan_samples(uint32_t B, uint32_t n) { return B * n * n < kPlanThreads ? B * n * n : kPlanThreads; }
__host__ __device__ inline PlanSample plan_sample(uint32_t i, uint32_t B, uint32_t n) {
    if (B * n * n <= kPlanThreads) return PlanSample{i / (n * n), i / n % n, i % n};
    // 2^32 times 1.2207440846057596 to the power of -1, -2 and -3; the products wrap, which takes the whole parts away
    auto coordinate = [i](uint32_t step, uint32_t size) {
        return static_cast<uint32_t>((static_cast<uint64_t>((i + 1u) * step) * size) >> 32);
    };
    return PlanSample{coordinate(3518319155u, B), coordinate(2882110345u, n), coordinate(2360945575u, n)};
}

// Which pair of query tiles looks through the K and V of a key tile that some pairs leave out and others work on: one that
// works on it, kNoChecker if none does or none leaves it out.  The first one from the diagonal on, so that every pair has
// about two key tiles of its own to look through, whatever the mask.  (Every pair next to one that leaves the tile out: with
// blocks of 256 x 128 of which half are -inf B=1 R=40 L=4096 H=128 took 253 us; 189 with K and V looked through by the plan.)
constexpr uint32_t kNoChecker = 0xFFFFu;
// cls: the classes of the key tile's tiles, `pitch` apart from query tile to query tile.
__host__ __device__ inline uint32_t plan_checker(const volatile uint8_t* cls, uint32_t pitch, uint32_t n, uint32_t kt) {
    const uint32_t q_pairs = (n + 1u) / 2u;
    uint32_t pair = kt / 2u, checker = kNoChecker;
    bool left_out = false;
#pragma unroll 4
    for (uint32_t d = 0; d < q_pairs; ++d) {
        const volatile uint8_t* at = cls + 2u * pair * pitch;
        const uint32_t x = *at, y = *(2u * pair + 1u < n ? at + pitch : at);
        if ((x | y) == kTileNeg) left_out = true;
        else if (checker == kNoChecker) checker = pair;
        pair = pair + 1u == q_pairs ? 0u : pair + 1u;
    }
    return left_out ? checker : kNoChecker;
}

// kCopy: the mask's rows start on no 16-byte boundary and are copied.  Else a kernel without a plan stands ready for a mask
// that leaves little out, and for K and V that items of the planned kernel find not to be finite.  grid: at most the launch
// bound's CTAs per SM.  The tiles of the mask round-robin, then a run of the parts of K and V; the CTA that is through last
// writes the lists, one group of 8, 16 or 32 lanes per pair of query tiles.
template <bool kCopy>
__global__ void __launch_bounds__(kPlanThreads, kCopy ? kPlanCopyCtasPerSm : kPlanCtasPerSm) fa_mask_plan(const PlanArgs args) {
    __shared__ uint32_t hist[kPlanMaxTiles + 1], cost[2];
    __shared__ uint16_t lens[kPlanMaxGroups], checkers[2 * kPlanMaxGroups];   // B n is at most twice the groups
    __shared__ bool last;
    __shared__ __align__(16) uint32_t staged[kPlanThreads / 32u * 16u * kPlanRowWords];
    grid_dep_wait();
    grid_dep_launch();
    PlanArgs a = args;   // (the inputs' addresses, for ld_settled)
    const uint32_t settled = zero_behind_the_wait();
    a.mask += settled, a.k += settled, a.v += settled;
    const uint32_t tid = threadIdx.x, n = a.n;
    // The first tile is on its way while the CTA finds out whether there is a plan, and looks at its parts of K and V.
    uint32_t* my_rows = staged + (tid >> 5) * (16u * kPlanRowWords);
    const uint32_t tiles = a.B * n * n;
    uint32_t tile = blockIdx.x;
    PlanRows rows = plan_rows(a, tile);
    if (tile < tiles) plan_fetch_tile<kCopy>(rows, my_rows);
    if (tile + gridDim.x < tiles) {   // the next one as far as L2: a row's 256 bytes per two lanes
        const PlanRows next = plan_rows(a, tile + gridDim.x);
        const uint32_t lane = tid & 31u, key = (lane & 1u) * 64u;
        if ((lane >> 1) < next.rows && key < next.keys) prefetch_l2(next.first + (lane >> 1) * next.pitch + 2u * key);
    }
    if constexpr (!kCopy) {
        // A tile that is -inf throughout begins with -inf.  Where fewer than a fifth of the tiles looked at do (and some of
        // them begins with neither -inf nor zero, or none with -inf), every CTA finds so for itself, nothing more is read
        // and the kernel without a plan takes the call.  One tile per thread is looked at (plan_sample): the 1024 of B=4
        // L=2048 took every CTA 5 us.
        const uint32_t of = plan_samples(a.B, n);
        uint32_t begins = 0;   // with -inf: 1, with zero: 1 << 16
        if (tid < of) {
            const PlanSample at = plan_sample(tid, a.B, n);
            const uint32_t v = ld_settled(reinterpret_cast<const uint16_t*>(a.mask) + (static_cast<size_t>(at.b) * a.L + at.qt * kTile) * a.L + at.kt * kTile);
            begins = v == 0xFC00u ? 1u : ((v & 0x7FFFu) == 0u ? 1u << 16 : 0u);
        }
        if (tid == 0) cost[0] = 0;
        __syncthreads();
        begins = __reduce_add_sync(0xffffffffu, begins);
        if ((tid & 31u) == 0) atomicAdd(&cost[0], begins);
        __syncthreads();
        const uint32_t neg = cost[0] & 0xFFFFu, zero = cost[0] >> 16;
        if (5u * neg < of && (neg == 0u || neg + zero < of)) {
            if (tid == 0 && blockIdx.x == 0) a.head[0] = 0;
            cp_async_wait_all();
            return;
        }
    }
    const uint32_t chunks = (a.F + kPlanCols - 1u) / kPlanCols, jobs = a.B * n * 2u * chunks;   // (launcher: below 2^31 / gridDim.x)
    uint32_t job = static_cast<uint32_t>(static_cast<uint64_t>(jobs) * blockIdx.x / gridDim.x);
    const uint32_t job_end = static_cast<uint32_t>(static_cast<uint64_t>(jobs) * (blockIdx.x + 1u) / gridDim.x);
    while (job < job_end) {   // parts of one key tile at a time (while the tile is on its way)
        const uint32_t bk = job / (2u * chunks), end = min(job_end, (bk + 1u) * 2u * chunks), b = bk / n, kt = bk % n;
        if (plan_looks_through<kCopy>(a, b, kt)) {
            for (; job < end; ++job) {
                const uint32_t part = job - bk * 2u * chunks;
                plan_finite(a, part < chunks ? a.k : a.v, b, kt, (part < chunks ? part : part - chunks) * kPlanCols);
            }
        }
        job = end;
    }
    while (tile < tiles) {
        plan_look_at_tile<kCopy>(a, rows, tile, my_rows);
        tile += gridDim.x;
        if (tile >= tiles) break;
        __syncwarp();   // every lane is through with these rows
        rows = plan_rows(a, tile);
        plan_fetch_tile<kCopy>(rows, my_rows);
    }
    __syncthreads();
    if (tid == 0) {   // (the barrier orders what the other threads wrote before this, the fence passes it on)
        __threadfence();
        last = atomicAdd(a.ticket, 1u) + 1u == gridDim.x;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    const uint32_t groups = a.B * a.q_pairs;
    const uint32_t width = n <= 8u ? 8u : (n <= 16u ? 16u : 32u), per_warp = 32u / width;
    const uint32_t lane = tid & 31u, sub = lane / width, l_in = lane % width;
    const uint32_t sub_mask = (width == 32u ? 0xFFFFFFFFu : (1u << width) - 1u) << (sub * width);
    // Where the lists (or plan_checker) take more than one step, each of which would wait for L2, the classes, and which K and V
    // are not finite, are brought into shared memory all at once, if they fit.  (All loops from here on stay loops: one CTA
    // goes through this code, once, and meets all of it for the first time.  Written out, and with what only the other
    // instance needs, the plan of B=8 R=12 L=387 H=16 causal took 9.8 us instead of 8.5, and the call of B=4 R=12 L=1021 H=64
    // 1 us more.)
    const uint8_t* cls = a.cls;
    const uint32_t* bad_of = a.bad;
    const uint32_t cls_words = (tiles + 3u) / 4u;   // (the bytes behind the classes are the scratch's own)
    if ((!kCopy || groups > kPlanThreads / 32u * per_warp || n > width) && cls_words + a.B * n <= sizeof(staged) / sizeof(uint32_t)) {
#pragma unroll 1
        for (uint32_t i = tid; i < cls_words; i += kPlanThreads) staged[i] = __ldcg(reinterpret_cast<const uint32_t*>(a.cls) + i);
#pragma unroll 1
        for (uint32_t i = tid; i < a.B * n; i += kPlanThreads) staged[cls_words + i] = __ldcg(a.bad + i);
        cls = reinterpret_cast<const uint8_t*>(staged);
        bad_of = staged + cls_words;
    }
#pragma unroll 1
    for (uint32_t i = tid; i <= n; i += kPlanThreads) hist[i] = 0;
    if (tid < 2) cost[tid] = 0;
    if (tid == 0) *a.ticket = 0;
    __syncthreads();
    if constexpr (!kCopy) {
        for (uint32_t i = tid; i < a.B * n; i += kPlanThreads)
            checkers[i] = static_cast<uint16_t>(plan_checker(cls + (i / n) * n * n + i % n, n, n, i % n));
        __syncthreads();
    }
    uint32_t mask_tiles = 0, steps = 0;
#pragma unroll 1
    for (uint32_t g0 = (tid >> 5) * per_warp; g0 < groups; g0 += kPlanThreads / 32u * per_warp) {
        const uint32_t gr = g0 + sub;
        const bool live = gr < groups;
        const uint32_t b = gr / a.q_pairs, q0 = (gr % a.q_pairs) * 2u;
        const volatile uint8_t* c0 = cls + (b * n + q0) * n;
        const bool two = q0 + 1u < n;   // the second query tile exists
        uint16_t* out = a.list + gr * n;
        uint32_t len = 0;
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < n; k0 += width) {
            const uint32_t kt = k0 + l_in;
            const bool in = live && kt < n;
            uint32_t x = kTileNeg, y = kTileNeg, bad = a.stamp + 1u;
            uint32_t checker = kNoChecker;
            if (in) {   // (all asked for together)
                const volatile uint8_t* c = c0 + kt;
                x = *c;
                bad = *const_cast<const volatile uint32_t*>(bad_of + b * n + kt);
                y = *(two ? c + n : c);
                if constexpr (!kCopy) checker = checkers[b * n + kt];
                if (!two) y = x == kTileNeg ? kTileNeg : kTileZero;
            }
            const bool keep = in && (x != kTileNeg || y != kTileNeg || bad == a.stamp);
            // (every head of the pair that looks a key tile through looks at its own columns)
            const uint32_t check = checker == gr % a.q_pairs && bad != a.stamp ? kStepCheck : 0u;
            const uint32_t votes = __ballot_sync(0xffffffffu, keep) & sub_mask;
            if (keep) {
                auto what = [](uint32_t c) { return c == kTileZero ? kStepNoMask : (c == kTileNeg ? kStepAllNeg : (c == kTileRows ? kStepRows : kStepMask)); };
                const uint32_t ex = what(x), ey = what(y);
                mask_tiles += (ex == kStepMask ? 1u : 0u) + (ey == kStepMask ? 1u : 0u);
                out[len + __popc(votes & ((1u << lane) - 1u))] = static_cast<uint16_t>(kt | check | (ex << kStepShift0) | (ey << kStepShift1));
            }
            len += __popc(votes);
        }
        if (live && l_in == 0) {
            if (len == 0) {   // nothing is left of these rows: one step with every key at -inf gives 0 / 0, as softmax does
                out[0] = static_cast<uint16_t>((kStepAllNeg << kStepShift0) | (kStepAllNeg << kStepShift1));
                len = 1;
            }
            lens[gr] = static_cast<uint16_t>(len);
            steps += len;
            atomicAdd(&hist[len], 1u);
        }
    }
    steps = __reduce_add_sync(0xffffffffu, steps);
    mask_tiles = __reduce_add_sync(0xffffffffu, mask_tiles);
    if (lane == 0) {
        atomicAdd(&cost[0], steps);
        atomicAdd(&cost[1], mask_tiles);
    }
    __syncthreads();
    if (tid == 0) {   // places, longest first
        uint32_t at = 0;
#pragma unroll 1
        for (uint32_t len = n; len >= 1u; --len) {
            const uint32_t c = hist[len];
            hist[len] = at;
            at += c;
        }
        // The planned kernel needs about 1.0 for a step and 0.2 more for each mask tile of it, the one without a plan
        // 1.2 for each step of all.
        *reinterpret_cast<const __half**>(a.head + kPlanInputs) = a.k;
        *reinterpret_cast<const __half**>(a.head + kPlanInputs + 2) = a.v;
        a.head[0] = kCopy || 5u * cost[0] + cost[1] < 6u * groups * n ? 1u : 0u;
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t gr = tid; gr < groups; gr += kPlanThreads)
        a.order[atomicAdd(&hist[lens[gr]], 1u)] = gr | (static_cast<uint32_t>(lens[gr]) << kPlanLenShift);
}

}  // namespace fa
