// What an additive mask leaves to do, found out once per call ahead of the attention kernel (fa_fwd_pipelined with
// kMaskPlanned).  The mask is shared by the heads, so one pass over it saves every head's pass over
//   - key tiles (128 keys) that the mask takes away from all 256 query rows of a work item: half of a causal mask,
//     the padding of a batch.  They are left out: P would be 0 there, so neither l nor O changes;
//   - the mask tiles that are zero throughout (nothing is added) or -inf throughout (no tile is fetched).
// A mask whose rows TMA cannot fetch (row starts on no 16-byte boundary) is copied on the way, the tiles that are
// neither, into rows that it can.
//
// Leaving a key tile out is only the same as adding -inf while its K and V are finite: 0 * inf and inf - inf are
// NaN.  So the K and V rows of every key tile that might be left out for some query tile are looked through as well,
// and a tile with an infinity or a NaN in it is not left out.  (Q need not be looked at: a row of Q with an infinity
// or a NaN has no finite score, so its result is NaN whatever is left out.)
#pragma once

#include "fa_kernels.cuh"

namespace fa {

struct PlanArgs {
    const __half* mask;    // [B, L, L]
    const __half* k;       // [B, L, F]
    const __half* v;
    __half* copy;          // [B, L, copy_pitch] or nullptr: rows that start on 16-byte boundaries
    uint8_t* cls;          // [B][n][n] (query tile, key tile): kTileNeg, kTileZero or kTileMixed
    uint32_t* head;        // {1 = the planned kernel runs, 0 = the one behind it}
    uint32_t* ticket;      // CTAs that are through; zero between launches
    uint32_t* bad;         // [B][n]: `stamp` if the key tile's K or V is not finite throughout
    uint32_t* order;       // [B * q_pairs]: (query pair of a batch entry) | key steps << kPlanLenShift, longest first
    uint16_t* list;        // [B * q_pairs][n]: key steps, see kStepShift0
    uint32_t B, L, F, n, q_pairs, copy_pitch;
    uint32_t stamp;           // of this call alone (a leftover that equals it costs a step, no more)
    uint32_t dense_allowed;   // a kernel without a plan stands ready for a mask that leaves little out
};
constexpr uint8_t kTileNeg = 0, kTileZero = 1, kTileMixed = 2;
constexpr uint32_t kPlanThreads = 256;
// CTAs per SM, 32 KB of loads in flight each; the instance that copies keeps a tile in registers, which fewer leave room for
// (B=4 R=12 L=1021 H=64, the whole call: 40.5 us with four, 39.2 with three, 40.8 with two).
constexpr uint32_t kPlanCtasPerSm = 4, kPlanCopyCtasPerSm = 3;
constexpr uint32_t kPlanCols = 128;         // columns of K or V that are looked through at a time
constexpr uint32_t kPlanMaxTiles = 256;     // key tiles per sequence,
constexpr uint32_t kPlanMaxGroups = 1024;   // and pairs of query tiles of all batch entries that the lists are built for

// One 128 x 128 tile of the mask: its class, and its copy.
template <bool kCopy>
__device__ __forceinline__ void plan_mask_tile(const PlanArgs& a, uint32_t tile) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t kt = tile % a.n, qt = (tile / a.n) % a.n, b = tile / (a.n * a.n);
    const uint32_t row0 = qt * kTile + warp * 16u, key0 = kt * kTile;
    const uint16_t* base = reinterpret_cast<const uint16_t*>(a.mask) + (static_cast<size_t>(b) * a.L + row0) * a.L + key0;
    const uint32_t rows = row0 < a.L ? min(16u, a.L - row0) : 0u;   // of this warp
    const uint32_t keys = min(kTile + 0u, a.L - key0);
    uint32_t not_neg = 0, not_zero = 0;
    // Rows on no 16-byte boundary: this warp's 16 rows in whole words where all of them, and a word more, lie inside the
    // mask (B=4 R=12 L=1021 H=64, the whole call 46 us with values one by one, 39 with words), else value by value.
    const uint64_t mask0 = reinterpret_cast<uint64_t>(a.mask), first = reinterpret_cast<uint64_t>(base), pitch = 2ull * a.L;
    const bool words = (first & ~3ull) >= mask0 && first + 15u * pitch + 260u <= mask0 + 2ull * a.B * a.L * a.L;
    uint32_t w[16][2], extra = 0;
    auto two_keys = [&](uint32_t r, uint32_t col) -> uint32_t {
        const uint16_t* at = base + static_cast<size_t>(r) * a.L + col;
        const uint32_t lo = r < rows && col < keys ? ld_settled(at) : 0u;
        const uint32_t hi = r < rows && col + 1u < keys ? ld_settled(at + 1) : 0u;
        return lo | (hi << 16);
    };
    // (four rows in flight together: one after the other, such a warp's way is what the whole plan waits for)
    auto four_rows = [&](uint32_t r0, uint32_t (&v)[4][2]) {
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) v[u][h] = two_keys(r0 + u, h * 64u + lane * 2u);
    };
    if constexpr (!kCopy) {   // rows on 16-byte boundaries: two rows a load, eight keys a lane (L is a multiple of 8)
        const uint32_t col = (lane & 15u) * 8u;
        uint4 x[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t r = 2u * i + (lane >> 4);
            if (r < rows && col < keys) x[i] = ld_settled(reinterpret_cast<const uint4*>(base + static_cast<size_t>(r) * a.L + col));
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t r = 2u * i + (lane >> 4);
            if (r < rows && col < keys) {
                not_neg |= (x[i].x ^ 0xFC00FC00u) | (x[i].y ^ 0xFC00FC00u) | (x[i].z ^ 0xFC00FC00u) | (x[i].w ^ 0xFC00FC00u);
                not_zero |= (x[i].x | x[i].y | x[i].z | x[i].w) & 0x7FFF7FFFu;
            }
        }
    } else if (words) {
        // Whole aligned words: word j of a row that starts in the middle of one holds its keys 2 j - 1 and 2 j.
#pragma unroll
        for (uint32_t r = 0; r < 16; ++r)
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h)
                w[r][h] = ld_settled(reinterpret_cast<const uint32_t*>((first + r * pitch) & ~3ull) + h * 32u + lane);
        extra = ld_settled(reinterpret_cast<const uint32_t*>((first + (lane & 15u) * pitch) & ~3ull) + 64);   // of row `lane`
#pragma unroll
        for (uint32_t r = 0; r < 16; ++r) {
            const uint32_t sh = static_cast<uint32_t>((first + r * pitch) >> 1) & 1u;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t lo = (h * 32u + lane) * 2u - sh;   // key of the low half (wraps below 0)
                const uint32_t valid = r < rows ? (lo < keys ? 0xFFFFu : 0u) | (lo + 1u < keys ? 0xFFFF0000u : 0u) : 0u;
                not_neg |= (w[r][h] ^ 0xFC00FC00u) & valid;
                not_zero |= w[r][h] & 0x7FFF7FFFu & valid;
            }
        }
        const uint32_t valid = lane < rows && ((first + lane * pitch) & 2u) != 0u && keys == kTile ? 0xFFFFu : 0u;   // key 127
        not_neg |= (extra ^ 0xFC00FC00u) & valid;
        not_zero |= extra & 0x7FFF7FFFu & valid;
    } else {
#pragma unroll 1
        for (uint32_t r0 = 0; r0 < rows; r0 += 4u) {
            uint32_t v[4][2];
            four_rows(r0, v);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t col = h * 64u + lane * 2u;
                    const uint32_t valid = r0 + u < rows ? (col + 1u < keys ? 0xFFFFFFFFu : (col < keys ? 0xFFFFu : 0u)) : 0u;
                    not_neg |= (v[u][h] ^ 0xFC00FC00u) & valid;
                    not_zero |= v[u][h] & 0x7FFF7FFFu & valid;
                }
        }
    }
    const bool any_not_neg = __syncthreads_or(not_neg != 0u), any_not_zero = __syncthreads_or(not_zero != 0u);
    if (tid == 0) a.cls[tile] = !any_not_neg ? kTileNeg : (any_not_zero ? kTileMixed : kTileZero);
    if constexpr (kCopy) {
        if (!any_not_neg || !any_not_zero) return;
        uint16_t* dst = reinterpret_cast<uint16_t*>(a.copy) + (static_cast<size_t>(b) * a.L + row0) * a.copy_pitch + key0;
        auto put = [&](uint32_t r, uint32_t h, uint32_t v) {
            const uint32_t col = h * 64u + lane * 2u;
            if (r < rows && col < keys)   // (the pitch is even: the second key has a place)
                *reinterpret_cast<uint32_t*>(dst + static_cast<size_t>(r) * a.copy_pitch + col) = v;
        };
        if (words) {
#pragma unroll
            for (uint32_t r = 0; r < 16; ++r) {   // the word behind each, from the next lane, and the two put together
                const uint32_t sh = (static_cast<uint32_t>((first + r * pitch) >> 1) & 1u) * 16u;
                const uint32_t n0 = __shfl_sync(0xffffffffu, w[r][0], (lane + 1u) & 31u), n1 = __shfl_sync(0xffffffffu, w[r][1], (lane + 1u) & 31u);
                const uint32_t head1 = __shfl_sync(0xffffffffu, w[r][1], 0), tail = __shfl_sync(0xffffffffu, extra, r);
                put(r, 0, __funnelshift_r(w[r][0], lane == 31u ? head1 : n0, sh));
                put(r, 1, __funnelshift_r(w[r][1], lane == 31u ? tail : n1, sh));
            }
        } else {
#pragma unroll 1
            for (uint32_t r0 = 0; r0 < rows; r0 += 4u) {
                uint32_t v[4][2];
                four_rows(r0, v);
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) put(r0 + u, h, v[u][h]);
            }
        }
    }
}

// Can any tile of the mask over key tile kt of batch entry b be -inf throughout?  Its first value tells when not.
__device__ __forceinline__ bool plan_maybe_left_out(const PlanArgs& a, uint32_t b, uint32_t kt) {
    bool neg = false;
    for (uint32_t qt = threadIdx.x; qt < a.n; qt += kPlanThreads)
        neg |= ld_settled(reinterpret_cast<const uint16_t*>(a.mask) + (static_cast<size_t>(b) * a.L + qt * kTile) * a.L + kt * kTile) == 0xFC00u;
    return __syncthreads_or(neg);
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
    for (uint32_t u = 0; u < 8; ++u)   // an exponent of all ones carries into the sign's place
        bits |= ((w[u].x & 0x7C007C00u) + 0x04000400u) | ((w[u].y & 0x7C007C00u) + 0x04000400u) |
                ((w[u].z & 0x7C007C00u) + 0x04000400u) | ((w[u].w & 0x7C007C00u) + 0x04000400u);
    if (bits & 0x80008000u) a.bad[b * a.n + kt] = a.stamp;
}

// kCopy: the mask's rows start on no 16-byte boundary and are copied.  grid: at most the launch bound's CTAs per SM.  The
// tiles of the mask round-robin, then a run of the parts of K and V; the CTA that is through last writes the lists, one
// group of 8, 16 or 32 lanes per pair of query tiles.
template <bool kCopy>
__global__ void __launch_bounds__(kPlanThreads, kCopy ? kPlanCopyCtasPerSm : kPlanCtasPerSm) fa_mask_plan(const PlanArgs args) {
    __shared__ uint32_t hist[kPlanMaxTiles + 1], cost[2];
    __shared__ uint16_t lens[kPlanMaxGroups];
    __shared__ bool last;
    grid_dep_wait();
    grid_dep_launch();
    PlanArgs a = args;   // (the inputs' addresses, for ld_settled)
    const uint32_t settled = zero_behind_the_wait();
    a.mask += settled, a.k += settled, a.v += settled;
    const uint32_t tid = threadIdx.x, n = a.n;
    if (a.dense_allowed) {
        // A tile that is -inf throughout begins with -inf.  Where fewer than a fifth of the tiles do, every CTA finds so
        // for itself, nothing more is read and the kernel without a plan takes the call.
        uint32_t neg = 0;
        for (uint32_t t = tid; t < a.B * n * n; t += kPlanThreads) {
            const uint32_t kt = t % n, qt = (t / n) % n, b = t / (n * n);
            neg += ld_settled(reinterpret_cast<const uint16_t*>(a.mask) + (static_cast<size_t>(b) * a.L + qt * kTile) * a.L + kt * kTile) == 0xFC00u;
        }
        if (tid == 0) cost[0] = 0;
        __syncthreads();
        neg = __reduce_add_sync(0xffffffffu, neg);
        if ((tid & 31u) == 0) atomicAdd(&cost[0], neg);
        __syncthreads();
        if (5u * cost[0] < a.B * n * n) {
            if (tid == 0 && blockIdx.x == 0) a.head[0] = 0;
            return;
        }
    }
    for (uint32_t t = blockIdx.x; t < a.B * n * n; t += gridDim.x) plan_mask_tile<kCopy>(a, t);
    const uint32_t chunks = (a.F + kPlanCols - 1u) / kPlanCols, jobs = a.B * n * 2u * chunks;   // (launcher: below 2^31 / gridDim.x)
    uint32_t job = static_cast<uint32_t>(static_cast<uint64_t>(jobs) * blockIdx.x / gridDim.x);
    const uint32_t job_end = static_cast<uint32_t>(static_cast<uint64_t>(jobs) * (blockIdx.x + 1u) / gridDim.x);
    while (job < job_end) {   // parts of one key tile at a time
        const uint32_t bk = job / (2u * chunks), end = min(job_end, (bk + 1u) * 2u * chunks), b = bk / n, kt = bk % n;
        if (plan_maybe_left_out(a, b, kt)) {
            for (; job < end; ++job) {
                const uint32_t part = job - bk * 2u * chunks;
                plan_finite(a, part < chunks ? a.k : a.v, b, kt, (part < chunks ? part : part - chunks) * kPlanCols);
            }
        }
        job = end;
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
    for (uint32_t i = tid; i <= n; i += kPlanThreads) hist[i] = 0;
    if (tid < 2) cost[tid] = 0;
    if (tid == 0) *a.ticket = 0;
    __syncthreads();
    const uint32_t width = n <= 8u ? 8u : (n <= 16u ? 16u : 32u), per_warp = 32u / width;
    const uint32_t lane = tid & 31u, sub = lane / width, l_in = lane % width;
    const uint32_t sub_mask = (width == 32u ? 0xFFFFFFFFu : (1u << width) - 1u) << (sub * width);
    uint32_t mask_tiles = 0, steps = 0;
    for (uint32_t g0 = (tid >> 5) * per_warp; g0 < groups; g0 += kPlanThreads / 32u * per_warp) {
        const uint32_t gr = g0 + sub;
        const bool live = gr < groups;
        const uint32_t b = gr / a.q_pairs, q0 = (gr % a.q_pairs) * 2u;
        const uint8_t* c0 = a.cls + (b * n + q0) * n;
        const bool two = q0 + 1u < n;   // the second query tile exists
        uint16_t* out = a.list + gr * n;
        uint32_t len = 0;
        for (uint32_t k0 = 0; k0 < n; k0 += width) {
            const uint32_t kt = k0 + l_in;
            const bool in = live && kt < n;
            uint32_t x = kTileNeg, y = kTileNeg, bad = a.stamp + 1u;
            if (in) {
                x = __ldcg(c0 + kt);
                bad = __ldcg(a.bad + b * n + kt);
                y = two ? __ldcg(c0 + n + kt) : (x == kTileNeg ? kTileNeg : kTileZero);
            }
            const bool keep = in && (x != kTileNeg || y != kTileNeg || bad == a.stamp);
            const uint32_t votes = __ballot_sync(0xffffffffu, keep) & sub_mask;
            if (keep) {
                const uint32_t ex = x == kTileZero ? kStepNoMask : (x == kTileNeg ? kStepAllNeg : kStepMask);
                const uint32_t ey = y == kTileZero ? kStepNoMask : (y == kTileNeg ? kStepAllNeg : kStepMask);
                mask_tiles += (ex == kStepMask ? 1u : 0u) + (ey == kStepMask ? 1u : 0u);
                out[len + __popc(votes & ((1u << lane) - 1u))] = static_cast<uint16_t>(kt | (ex << kStepShift0) | (ey << kStepShift1));
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
        for (uint32_t len = n; len >= 1u; --len) {
            const uint32_t c = hist[len];
            hist[len] = at;
            at += c;
        }
        // The planned kernel needs about 1.0 for a step and 0.2 more for each mask tile of it, the one without a plan
        // 1.2 for each step of all.
        a.head[0] = !a.dense_allowed || 5u * cost[0] + cost[1] < 6u * groups * n ? 1u : 0u;
    }
    __syncthreads();
    for (uint32_t gr = tid; gr < groups; gr += kPlanThreads)
        a.order[atomicAdd(&hist[lens[gr]], 1u)] = gr | (static_cast<uint32_t>(lens[gr]) << kPlanLenShift);
}

}  // namespace fa
