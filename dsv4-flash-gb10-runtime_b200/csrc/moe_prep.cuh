// What the batched routed-expert layer's kernels share: tile widths, work descriptors, the three-term MXFP4 quantiser; and its
// small kernels behind the GEMMs, the per-token sum and the expert-parallel exchange (grouping and activations:
// moe_prep_kernel.cuh).
#pragma once

#include "gemv_engine.cuh"

namespace dsv4 {

constexpr int kMoeMaxExperts = 1024;
constexpr int kMoeTileRows = 128;      // weight rows per tensor-core tile (the MMA's M)
constexpr int kMoeTileTokens = 128;    // tokens per tile at most, fp16 path

// The tokens of a tile are padded to one of seven column counts (the boxes the activation copies are encoded for): a multiple of 16, or
// all that a tile may have.  (48 and 80 among them: 256 experts of 4096, 2048, top 6, 1 800 tokens 724 -> 692 us, 2 800 tokens 824 -> 795.)
constexpr int kMoeWidths = 7;
__host__ __device__ __forceinline__ int moe_width_index(int n) { return n <= 16 ? 0 : n <= 96 ? (n - 1) >> 4 : 6; }
__host__ __device__ __forceinline__ int moe_width(int index, int cap) { return index == 6 ? cap : 16 * (index + 1); }
// The n tokens of an expert are cut into the fewest tiles of at most `cap`, all but the last of one size: tiles of one
// size finish together.
__host__ __device__ __forceinline__ int moe_token_tiles(int n, int cap) { return (n + cap - 1) / cap; }
__host__ __device__ __forceinline__ int moe_tokens_per_tile(int n, int cap) {
    const int nt = moe_token_tiles(n, cap);
    return nt == 0 ? cap : moe_width(moe_width_index((n + nt - 1) / nt), cap);
}

// Work descriptors written by the grouping kernel, read by the kernels after it.
struct MoeGroups {
    int* offsets;        // [E + 1] first slot of every expert (slots = pairs sorted by expert)
    int* tiles_up;       // [E + 1] prefix sum of gate/up tiles per expert
    int* tiles_down;     // [E + 1] prefix sum of down tiles per expert
    int* pair_slot;      // [P] pair index -> slot, -1 for a dropped pair
    float* slot_w;       // [P] router weight of a slot
};

// out[t, :] = bf16( sum_j y[slot(t, j), :] ), j in the router's order (fixed summation order).
__global__ void moe_combine_kernel(const float* __restrict__ y, const int* __restrict__ pair_slot, int n_tokens,
                                   int k, int O, __nv_bfloat16* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    const int o = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (o >= O) return;
    for (int t = blockIdx.y; t < n_tokens; t += gridDim.y) {         // grid.y is capped at 65 535
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < k; ++j) {
            const int slot = pair_slot[t * k + j];
            if (slot < 0) continue;
            const float4 v = __ldcs(reinterpret_cast<const float4*>(y + (size_t)slot * O + o));
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
        uint2 packed;
        packed.x = *reinterpret_cast<uint32_t*>(&lo);
        packed.y = *reinterpret_cast<uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(out + (size_t)t * O + o) = packed;
    }
}

// Expert parallel: where the per-token sums of a rank go.  Token t of the gathered batch belongs to rank
// t / tokens_per_rank; its partial row is stored straight into THAT rank's receive buffer (a peer pointer: plain
// stores over NVLink, no collective), at [my_rank][t % tokens_per_rank][O].
constexpr int kMoeMaxRanks = 16;
struct MoePeerOut {
    __nv_bfloat16* recv[kMoeMaxRanks];     // receive buffer of every rank, [world][tokens_per_rank][O] bf16
    int world, my_rank, tokens_per_rank;
};

// Expert parallel, input side: the tokens of the gathered batch are not copied together first; rank r's tokens
// are read where they are, from the buffers rank r published (peer pointers: plain loads over NVLink).
struct MoePeerIn {
    const __nv_bfloat16* x[kMoeMaxRanks];      // [tokens_per_rank, K] bf16 of every rank
    const int* ids[kMoeMaxRanks];              // [tokens_per_rank, k] GLOBAL expert ids
    const float* w[kMoeMaxRanks];              // [tokens_per_rank, k] router weights
    int world, my_rank, tokens_per_rank, experts_per_rank;
};

// ids / weights of all ranks -> this rank's view of the gathered batch: local expert index, or -1 where the
// expert lives on another rank (a pair the layer skips).
__global__ void moe_ep_gather_meta_kernel(const MoePeerIn in, int k, int* __restrict__ ids_local,
                                          float* __restrict__ w_local) {
    pdl_launch_dependents();
    pdl_wait();
    const int per_rank = in.tokens_per_rank * k;
    const int n = in.world * per_rank;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int r = i / per_rank, j = i - r * per_rank;
        const int e = __ldcg(in.ids[r] + j) - in.my_rank * in.experts_per_rank;
        ids_local[i] = (e >= 0 && e < in.experts_per_rank) ? e : -1;
        w_local[i] = __ldcg(in.w[r] + j);
    }
}

// moe_combine_kernel with the peer destination above: the exchange is the kernel's own stores, row by row.
__global__ void moe_combine_peer_kernel(const float* __restrict__ y, const int* __restrict__ pair_slot, int n_tokens,
                                        int k, int O, const MoePeerOut peer) {
    pdl_launch_dependents();
    pdl_wait();
    const int o = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (o >= O) return;
    for (int t = blockIdx.y; t < n_tokens; t += gridDim.y) {         // grid.y is capped at 65 535
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        bool any = false;
        for (int j = 0; j < k; ++j) {
            const int slot = pair_slot[t * k + j];
            if (slot < 0) continue;
            any = true;
            const float4 v = __ldcs(reinterpret_cast<const float4*>(y + (size_t)slot * O + o));
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        if (!any) continue;                 // none of the token's experts lives here: the home rank skips this slice
        __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
        uint2 packed;
        packed.x = *reinterpret_cast<uint32_t*>(&lo);
        packed.y = *reinterpret_cast<uint32_t*>(&hi);
        const int home = t / peer.tokens_per_rank, tl = t - home * peer.tokens_per_rank;
        __nv_bfloat16* dst = peer.recv[home] + ((size_t)peer.my_rank * peer.tokens_per_rank + tl) * O + o;
        *reinterpret_cast<uint2*>(dst) = packed;
    }
}

// out[t, :] = bf16( sum_r recv[r][t, :] ), ranks in ascending order (fixed summation order), over the ranks that
// own at least one of the token's experts (ids [n_tokens, k] global, experts_per_rank per rank): the others wrote
// nothing.
__global__ void moe_ep_sum_kernel(const __nv_bfloat16* __restrict__ recv, const int* __restrict__ ids, int k,
                                  int experts_per_rank, int world, int n_tokens, int O,
                                  __nv_bfloat16* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t n4 = (size_t)n_tokens * O / 4;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        const int t = (int)(i / (size_t)(O / 4));
        uint32_t owners = 0;
        for (int j = 0; j < k; ++j) {
            const int e = ids[t * k + j];
            if (e >= 0 && e / experts_per_rank < world) owners |= 1u << (e / experts_per_rank);
        }
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < world; ++r) {
            if (!((owners >> r) & 1u)) continue;
            const uint2 q = __ldcs(reinterpret_cast<const uint2*>(recv + (size_t)r * n_tokens * O) + i);
            acc.x += __uint_as_float(q.x << 16); acc.y += __uint_as_float(q.x & 0xffff0000u);
            acc.z += __uint_as_float(q.y << 16); acc.w += __uint_as_float(q.y & 0xffff0000u);
        }
        __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
        uint2 packed;
        packed.x = *reinterpret_cast<uint32_t*>(&lo);
        packed.y = *reinterpret_cast<uint32_t*>(&hi);
        reinterpret_cast<uint2*>(out)[i] = packed;
    }
}

// Eight neighbouring elements per lane, four lanes per 32-element block -> three MXFP4 terms whose sum reproduces the
// block to ~11 bits:
//   v ~ q1 * 2^e1 + q2 * 2^e2 + q3 * 2^e3,  q E2M1, 2^e the smallest power of two with amax(what is left) <= 6 * 2^e
// (no saturation), each term the round-to-nearest E2M1 quantisation of the residual the previous terms left.  The tensor
// cores multiply FP4 by FP4; three terms are what keeps the layer inside its tolerance (one term: cosine 0.993).
// word[t]: the lane's eight packed elements of term t; scale[t]: the block's E8M0 byte (in all four lanes).
__device__ __forceinline__ void moe_quantize_mxfp4x3(float (&v)[8], uint32_t (&word)[3], uint32_t (&scale)[3]) {
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
        m = max(m, __shfl_xor_sync(kFullMask, m, 1));
        m = max(m, __shfl_xor_sync(kFullMask, m, 2));
        int e = (int)((m + 0x003fffffu) >> 23) - 129;               // above 6 * 2^e the E2M1 grid would saturate
        e = min(max(e, -127), 127);
        const float inv = __uint_as_float((uint32_t)min(max(127 - e, 1), 254) << 23);
        const float sc = __uint_as_float((uint32_t)max(e + 127, 1) << 23);                     // 2^e (>= 2^-126)
        word[t] = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint16_t packed;
            asm("{\n .reg .b8 b;\n cvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n mov.b16 %0, {b, 0};\n}"
                : "=h"(packed) : "f"(v[2 * i] * inv), "f"(v[2 * i + 1] * inv));
            if (t < 2) {
                const float2 back = e2m1x2_to_float2(packed);
                v[2 * i] = fmaf(-back.x, sc, v[2 * i]);
                v[2 * i + 1] = fmaf(-back.y, sc, v[2 * i + 1]);
            }
            word[t] |= (uint32_t)(packed & 0xff) << (8 * i);
        }
        scale[t] = (uint32_t)(e + 127);
    }
}

// The same of a whole block by one lane.
__device__ __forceinline__ void moe_quantize_block_x3(float (&v)[32], uint4 (&word)[3], uint32_t (&scale)[3]) {
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
        int e = (int)((m + 0x003fffffu) >> 23) - 129;
        e = min(max(e, -127), 127);
        const float inv = __uint_as_float((uint32_t)min(max(127 - e, 1), 254) << 23);
        const float sc = __uint_as_float((uint32_t)max(e + 127, 1) << 23);
        uint32_t r[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            uint16_t packed;
            asm("{\n .reg .b8 b;\n cvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n mov.b16 %0, {b, 0};\n}"
                : "=h"(packed) : "f"(v[2 * i] * inv), "f"(v[2 * i + 1] * inv));
            if (t < 2) {
                const float2 back = e2m1x2_to_float2(packed);
                v[2 * i] = fmaf(-back.x, sc, v[2 * i]);
                v[2 * i + 1] = fmaf(-back.y, sc, v[2 * i + 1]);
            }
            r[i >> 2] |= (uint32_t)(packed & 0xff) << (8 * (i & 3));
        }
        word[t] = make_uint4(r[0], r[1], r[2], r[3]);
        scale[t] = (uint32_t)(e + 127);
    }
}

// 16 elements of a 32-element block whose largest magnitude is m (float bits) -> three E4M3 terms,
//   v ~ 2^e (q1 + 2^-4 q2 + 2^-(4 + STEP) q3),   2^e such that the largest q1 is in [128, 256),
// each term rounding what the ones before it left: a term takes four significant bits and leaves at most half a step of its last, so the
// next in units 16 times smaller is below 256.  STEP = kE4m3MidStep (FP32 values): 11 bits and more of an element down to 2^-13 of the
// block's largest.  STEP = kE4m3BfStep (bf16 values): two terms hold such an element exactly, and the third is kept for smaller ones, whose
// first two terms are subnormal: exact down to 2^-18 of the block's largest, four bits far below.
// A block with an infinity or a NaN gets scale byte 0xFF, E8M0's NaN.
constexpr int kE4m3MidStep = 4, kE4m3BfStep = 14;
template <int STEP>
__device__ __forceinline__ void moe_quantize_e4m3x3(float (&v)[16], uint32_t m, uint4 (&packed)[3], uint32_t (&scale)[3]) {
    const int e = max((int)(m >> 23) - 7, 4 + STEP + 2);                    // biased
    const bool finite = m < 0x7f800000u;
    const float inv = __uint_as_float((uint32_t)max(254 - e, 1) << 23);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= inv;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        uint32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t half[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float &lo = v[4 * i + 2 * j], &hi = v[4 * i + 2 * j + 1];
                uint16_t q;
                asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(q) : "f"(hi), "f"(lo));
                half[j] = q;
                if (t < 2) {
                    uint32_t h;
                    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"(q));
                    const float2 back = __half22float2(*reinterpret_cast<const __half2*>(&h));
                    const float up = t == 0 ? 16.f : (float)(1 << STEP);
                    lo = (lo - back.x) * up;
                    hi = (hi - back.y) * up;
                }
            }
            r[i] = half[0] | (half[1] << 16);
        }
        packed[t] = make_uint4(r[0], r[1], r[2], r[3]);
        scale[t] = finite ? (uint32_t)(t == 0 ? e : t == 1 ? e - 4 : e - 4 - STEP) : 255u;
    }
}

}  // namespace dsv4
