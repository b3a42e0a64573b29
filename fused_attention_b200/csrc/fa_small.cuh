// Fused attention forward for short sequences (at most 160 keys): many small problems, such as attention inside the
// windows of an image.
//
// Why not the tcgen05 kernels: their tile is 128 query rows, of which a window of 49 uses 49 (and 128 x 128 scores of
// which 49 x 49), and a CTA sets up barriers, tensor memory and descriptors for one such tile.  What bounds these calls
// is neither the products nor the exponentials but memory and the latency of a chain of load, product, softmax,
// product, store per problem; so a CTA here is small (a warp per 16 query rows, warp-wide mma.sync with the scores of a
// row in registers, no state but its tiles in shared memory) and up to a dozen of them per SM hide one another's chain.
// All keys are there at once: one pass, no running maximum.  Same arithmetic as the other kernels: fp16 operands, fp32
// scores, maximum, sum and numerator, exp2 with log2(e)/sqrt(H) folded in, P rounded to fp16.
// Measured, B=256 R=8 L=49 H=32 (27 MB with a mask): 29 us on the one-tile kernel and 44 with a mask, 7.4 and 10.8 here;
// B=1024 R=8 L=64 H=64 135 and 45 us (5.9 TB/s).
//
// The mask of a batch entry, L x L values that start anywhere, comes in as one run of words beside K and V.
#pragma once

#include "fa_ptx.cuh"

namespace fa {

struct SmallArgs {
    const __half* q;      // [B, L, F]
    const __half* k;
    const __half* v;
    const __half* mask;   // [B, L, L] or nullptr
    __half* y;
    uint32_t B, L, F, R;
    float scale_log2, mask_to_score;   // as in Params
};

template <int H, int KT>   // KT: 16-row tiles of queries and of keys
struct SmallCfg {
    static constexpr uint32_t kRows = KT * 16;
    static constexpr uint32_t kPitch = H * 2 + 16;   // bytes; eight rows of 16 bytes lie in different banks
    static constexpr uint32_t kTileBytes = kRows * kPitch;
    static constexpr uint32_t smem_bytes(uint32_t L, bool mask) {
        return 3u * kTileBytes + (mask ? ((2u * L * L + 2u * kRows + 4u + 15u) & ~15u) : 0u);
    }
};

template <int H, int KT, bool kHasMask>
__global__ void __launch_bounds__(KT * 32) fa_fwd_small(const SmallArgs a) {
    using C = SmallCfg<H, KT>;
    constexpr uint32_t kThreads = KT * 32;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t head = blockIdx.x % a.R, batch = blockIdx.x / a.R, L = a.L;
    const uint32_t sQ = smem_u32(smem_raw), sK = sQ + C::kTileBytes, sV = sK + C::kTileBytes, sM = sV + C::kTileBytes;
    grid_dep_wait();
    grid_dep_launch();

    // ---- Q, K, V (rows beyond the sequence as zeros) and the mask into shared memory
    const size_t at = static_cast<size_t>(batch) * L * a.F + head * H;
    constexpr uint32_t kVecs = H / 8;   // 16-byte pieces per row
    auto load = [&](uint32_t dst, const __half* src) {
#pragma unroll
        for (uint32_t i = tid; i < C::kRows * kVecs; i += kThreads) {
            const uint32_t r = i / kVecs, c = i % kVecs;
            cp_async_16_zero(dst + r * C::kPitch + c * 16u, src + at + static_cast<size_t>(r < L ? r : 0u) * a.F + c * 8u, r < L);
        }
    };
    load(sQ, a.q);
    load(sK, a.k);
    uint32_t mask_at = 0;   // the mask's first value in shared memory
    if constexpr (kHasMask) {
        const uint64_t base = reinterpret_cast<uint64_t>(a.mask), end = base + 2ull * a.B * L * L;
        const uint64_t first = base + 2ull * batch * L * L, bytes = 2ull * L * L;
        if (((first | bytes) & 15u) == 0u) {
            mask_at = sM;
            for (uint32_t i = tid * 16u; i < bytes; i += kThreads * 16u)
                cp_async_16_zero(sM + i, reinterpret_cast<const void*>(first + i), true);
        } else {
            const uint64_t start = first & ~3ull;
            const uint32_t lead = static_cast<uint32_t>(first - start);   // 0 or 2 bytes
            mask_at = sM + lead;
            for (uint32_t i = tid * 4u; i < lead + bytes; i += kThreads * 4u) {
                const uint64_t src = start + i;
                if (src >= base && src + 4u <= end) cp_async_4(sM + i, src);
                else if (src < base) st_shared_u16(sM + i + 2u, *reinterpret_cast<const uint16_t*>(src + 2u));
                else st_shared_u16(sM + i, *reinterpret_cast<const uint16_t*>(src));
            }
        }
    }
    cp_async_commit();
    load(sV, a.v);
    cp_async_commit();
    cp_async_wait_group<1>();   // all but V
    __syncthreads();

    // ---- this warp's 16 query rows: rows g and g + 8 of them in a lane
    const uint32_t row0 = warp * 16u, g = lane >> 2, t = lane & 3u;
    float s[KT * 2][4];
#pragma unroll
    for (int n = 0; n < KT * 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < H / 16; ++ks) {
        uint32_t qa[4];
        ldmatrix_x4(qa, sQ + (row0 + (lane & 15u)) * C::kPitch + ks * 32 + (lane >> 4) * 16u);
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) {
            uint32_t kb[4];
            ldmatrix_x4(kb, sK + (kt * 16 + (lane & 7u) + ((lane >> 4) << 3)) * C::kPitch + ks * 32 + ((lane >> 3) & 1u) * 16u);
            mma_m16n8k16(s[2 * kt], qa, kb[0], kb[1]);
            mma_m16n8k16(s[2 * kt + 1], qa, kb[2], kb[3]);
        }
    }
    if constexpr (kHasMask) {
        const uint32_t r0 = min(row0 + g, L - 1u), r1 = min(row0 + g + 8u, L - 1u);
        const uint32_t m0 = mask_at + (r0 * L + 2u * t) * 2u, m1 = mask_at + (r1 * L + 2u * t) * 2u;
        // (a key beyond the end reads on into the next row, and is taken out below)
        if (((2u * L | mask_at) & 3u) == 0u) {   // every row starts on a word
#pragma unroll
            for (int n = 0; n < KT * 2; ++n) {
                const uint32_t w0 = ld_shared_u32(m0 + n * 16), w1 = ld_shared_u32(m1 + n * 16);
                const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&w0));
                const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&w1));
                s[n][0] = fmaf(f0.x, a.mask_to_score, s[n][0]);
                s[n][1] = fmaf(f0.y, a.mask_to_score, s[n][1]);
                s[n][2] = fmaf(f1.x, a.mask_to_score, s[n][2]);
                s[n][3] = fmaf(f1.y, a.mask_to_score, s[n][3]);
            }
        } else {
#pragma unroll
            for (int n = 0; n < KT * 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    s[n][e] = fmaf(ld_shared_half(m0 + n * 16 + e * 2), a.mask_to_score, s[n][e]);
                    s[n][2 + e] = fmaf(ld_shared_half(m1 + n * 16 + e * 2), a.mask_to_score, s[n][2 + e]);
                }
        }
    }
#pragma unroll
    for (int n = 0; n < KT * 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (n * 8 + 2 * t + e >= L) s[n][e] = s[n][2 + e] = -INFINITY;
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < KT * 2; ++n) {
        mx0 = max3(mx0, s[n][0], s[n][1]);
        mx1 = max3(mx1, s[n][2], s[n][3]);
    }
#pragma unroll
    for (int d = 1; d <= 2; d <<= 1) {
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, d));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, d));
    }
    // (a row masked out completely takes 0 as its reference: P = 0, l = 0, and 0 / 0 as softmax gives)
    const float n0 = mx0 == -INFINITY ? 0.f : -mx0 * a.scale_log2, n1 = mx1 == -INFINITY ? 0.f : -mx1 * a.scale_log2;
    float l0 = 0.f, l1 = 0.f;
    uint32_t p[KT * 2][2];
#pragma unroll
    for (int n = 0; n < KT * 2; ++n) {
        const float p0 = ex2_approx(fmaf(s[n][0], a.scale_log2, n0)), p1 = ex2_approx(fmaf(s[n][1], a.scale_log2, n0));
        const float p2 = ex2_approx(fmaf(s[n][2], a.scale_log2, n1)), p3 = ex2_approx(fmaf(s[n][3], a.scale_log2, n1));
        l0 += p0 + p1;
        l1 += p2 + p3;
        p[n][0] = pack_half2(p0, p1);
        p[n][1] = pack_half2(p2, p3);
    }
#pragma unroll
    for (int d = 1; d <= 2; d <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, d);
        l1 += __shfl_xor_sync(0xffffffffu, l1, d);
    }
    cp_async_wait_group<0>();
    __syncthreads();   // V is there
    float o[H / 8][4];
#pragma unroll
    for (int n = 0; n < H / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        const uint32_t pa[4] = {p[2 * kt][0], p[2 * kt][1], p[2 * kt + 1][0], p[2 * kt + 1][1]};
#pragma unroll
        for (int d = 0; d < H / 16; ++d) {
            uint32_t vb[4];
            ldmatrix_x4_trans(vb, sV + (kt * 16 + (lane & 15u)) * C::kPitch + d * 32 + (lane >> 4) * 16u);
            mma_m16n8k16(o[2 * d], pa, vb[0], vb[1]);
            mma_m16n8k16(o[2 * d + 1], pa, vb[2], vb[3]);
        }
    }
    // ---- Y = O / l: through this warp's own rows of Q in shared memory, so that rows leave in 16-byte pieces
    const float i0 = 1.f / l0, i1 = 1.f / l1;
    const uint32_t y0 = sQ + (row0 + g) * C::kPitch + t * 4u, y1 = y0 + 8u * C::kPitch;
#pragma unroll
    for (int n = 0; n < H / 8; ++n) {
        st_shared_u32(y0 + n * 16, pack_half2(o[n][0] * i0, o[n][1] * i0));
        st_shared_u32(y1 + n * 16, pack_half2(o[n][2] * i1, o[n][3] * i1));
    }
    __syncwarp();
#pragma unroll
    for (uint32_t i = lane; i < 16u * kVecs; i += 32u) {
        const uint32_t r = i / kVecs, c = i % kVecs;
        if (row0 + r < L) {
            uint32_t w[4];
            ld_shared_v4(sQ + (row0 + r) * C::kPitch + c * 16u, w);
            *reinterpret_cast<uint4*>(a.y + at + static_cast<size_t>(row0 + r) * a.F + c * 8u) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

}  // namespace fa
