// Batched routed-expert GEMMs on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory): what the
// two tensor-core paths share, and the number formats of the path "fp16".
//
// For every expert e with its n_e tokens (pairs sorted by expert, "slots"):
//   up   : G[h, t] = W1_e[h, :] . x_t,  U[h, t] = W3_e[h, :] . x_t,  mid[slot, h] = silu(G) * U
//   down : y[slot, o] = w_pair * W2_e[o, :] . mid[slot, :]
// Weights are the MMA's A operand (M = 128 weight rows per tile), tokens its B operand (N = 16 .. 128 tokens),
// so a weight tile is read from HBM and dequantised ONCE for all tokens of the tile.
//
// Numbers of the path "fp16", two forms of it.  Products are exact and sums FP32 in both.
// (a) Block-scaled MMAs (moe_gemm_mxf4.cuh, MoeQFp8), up to kQMostTokensFp8 pairs per expert.
//   * weights: E2M1 with their scale bytes, exact (0xFF counts as 2^-127).
//   * x and the intermediate: three E4M3 terms with a scale per 32 elements (moe_quantize_e4m3x3), x exact down to 2^-18 of the largest of
//     its 32, the intermediate 11 bits and more down to 2^-13 of the largest of its 32.
//   * range: a token's x that is large or small, and an expert's W1 and W3 that are, are normalised (moe_act_fp8_kernel) and the powers of two
//     multiplied back in the epilogues; a product silu(G) * U beyond FP32 even so is the largest FP32 value.
//   * a token with an infinity or a NaN gives NaN throughout ((b): a mix of NaN, infinities and finite values).
//   Error beside the bf16 output's rounding, against 64 bits: 1.4e-5 of the norm, and 3.4e-5 with one channel of x in 32 a factor 2^14 larger
//   and its weights zero; (b) has 2.1e-4 and 8e-2.  One channel of the intermediate in 32 a factor 2^f larger: 5e-6 for any f, where (b) has
//   1.5e-4 at f = 6 and, saturating, 0.4 at f = 8 and 0.9 from 12 on; with its weights in W2 zero, so that only the others count, 1.1e-4 at f = 12,
//   2.3e-4 at 13, 1.5e-3 at 16 and 1.7e-2 at 20, where (b) stays at 2.0e-4: beyond 2^13 the smaller ones of 32 have fewer bits here.
// (b) fp16 MMAs (moe_gemm_kernel.cuh): more tokens, rows of other ranks, weights that are 16- but not 32-byte aligned, and shapes where (a)'s
//   operands have no room in the workspace (its x lies in the bytes of y, which is written when x is done with).
// Of (b):
//   * weights: E2M1 * 2^(s - c_row), c_row = largest E8M0 byte of the row.  E2M1 times a power of two is exact in fp16
//     down to 2^-24, i.e. blocks up to 2^23 times smaller than the row's largest are exact, smaller ones vanish; scale
//     byte 0xFF contributes 0.
//   * activations: x_t * 2^-e_t with the token's largest magnitude in [1, 2); q_t = floor(log2(rms)) of the result.
//   * mid is stored in fp16 as silu(G) * U * 2^-(2 (e_t + q_t) + c1 + c3 - 254 + L), c1 / c3 the expert's typical W1 / W3
//     scale byte and L = log2(K) + 2: a dot product of K values of a typical weight row (E2M1, rms about 2) with a token of
//     rms 1 is about 2 sqrt(K), so what is stored is of the order of 1 whatever the scales of x and of the weights, and
//     11 bits are kept over the nine orders of magnitude of fp16 around it.
// The powers of two are multiplied back in the epilogues, in FP32.
#pragma once

#include "moe_prep.cuh"
#include "stream_ring.cuh"
#include "tc05.cuh"

#include <cuda.h>

namespace dsv4 {

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_one(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// A value beyond the FP32 range (an infinity) as the largest in it; NaN stays.
__device__ __forceinline__ float saturate_finite(float v) {
    asm("min.NaN.f32 %0, %0, 0f7F7FFFFF;\n max.NaN.f32 %0, %0, 0fFF7FFFFF;" : "+f"(v));
    return v;
}

// 2^e as float for |e| well inside the FP32 range.
__device__ __forceinline__ float float_pow2(int e) {
    e = min(max(e, -126), 127);
    return __uint_as_float((uint32_t)(e + 127) << 23);
}

}  // namespace dsv4
