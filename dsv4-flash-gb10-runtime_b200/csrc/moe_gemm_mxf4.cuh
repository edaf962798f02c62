// Batched routed-expert GEMMs with BLOCK-SCALED tensor-core MMAs (tcgen05 kind::mxf4, UE8M0 scales in tensor
// memory): the MXFP4 weights go from HBM to shared memory to the tensor cores exactly as the checkpoint stores them
// (packed nibbles + E8M0 bytes) - no dequantisation instruction is executed, and a weight costs half a byte of
// shared-memory traffic.
//
// The tensor cores multiply FP4 by FP4, so the activations are given as three MXFP4 terms (moe_prep.cuh):
//   D = W * (q1 + q2 + q3) = W q1 + W q2 + W q3.
// Tiles: two blocks of 256 weight rows (rows m0.. of W1 and of W3 for gate/up, rows m0.. and m0 + 256.. of W2 for down)
// x up to 112 tokens, one tile per PAIR of CTAs (cta_group::2): each CTA holds 128 rows of both blocks and half of the
// tokens.  A stage covers 256 K-elements (one 128-byte swizzled row per operand row = 4 MMAs of K = 64).
//
// How the terms are multiplied.  Each term is an MMA of its own into the SAME accumulator columns, with the weight tile
// kept in the collector between the three: 3 x N / 2 clocks for N tokens (N >= 96), the full rate of the tensor pipe;
// a stage's 24 MMAs and 10 scale copies take 1 170 clocks at N = 96 and 580 at N = 16.  Without the collector every MMA
// reads its A tile again, 32 clocks at 128 bytes a clock.  Two accumulator sets of 2 x 112 columns fit into tensor memory,
// so the MMAs of a tile run while the one before it is read out.  (E4M3 tiles of few tokens: the three terms lie side by side
// along N, a third of the MMAs, 44 to 56 clocks each.  FP4 tiles that way were slower, 64 tokens 428 -> 458 us.)
//
// What bounds it: the weights.  A CTA takes in 34 KB of weights and scales per stage, 1 400 clocks of its share of 7 TB/s,
// so everything else has to keep out of the way of that stream, above all instruction issue: with six roles on a CTA an
// instruction of a single-thread role takes tens of clocks, not four.  Hence few instructions per stage: ONE producer
// thread with three copies (two weight boxes, one box with the three terms of the CTA's tokens - the rows of a tile are
// neighbours in memory, in slot order), ONE full and ONE empty barrier.  Gathering token rows four at a time instead took
// 36 copies per stage and held the stream at 4.6 TB/s.  Why pairs: they halve the activations a CTA takes in.
//
// CTA = 24 warps, persistent grid, one CTA per SM, tiles by static striding over the pairs:
//   warp 0        (CTA 0, one thread) scale atoms -> tensor memory, MMAs of the pair
//   warp 1        producer (one thread)
//   warps 4..15   epilogue: accumulators -> SwiGLU -> three MXFP4 terms (gate/up), or -> FP32 rows (down)
//   warps 16..23  scale bytes of weights and activations -> 512-byte scale atoms in shared memory; two groups of four warps
//                 take pairs of stages in turn, their loads a pair ahead, across tiles
// With one group of scale warps (busy 1 200 clocks per stage) and eight epilogue warps (1 100) the two of them, not the MMAs,
// set the pace: 1 700 clocks per stage of gate/up and 2 170 of down, whose tiles are half as long.
// The full barriers are CTA 0's: copies and scale warps of both CTAs arrive there.  The "empty" and "accumulator full"
// barriers are signalled in both CTAs by the commits.
// No operand passes through a register.
// Every wait is bounded; a CTA that gives up has polled far longer than any copy takes, so nothing is in flight when it
// leaves, and both CTAs meet at a cluster barrier before they exit.
#pragma once

#include "moe_gemm.cuh"

#include <type_traits>

namespace dsv4 {

// How the operands are held.  A stage is one 128-byte swizzled row per operand row, four MMAs.
//
// FP8 is the form of the path "fp16" (moe_gemm.cuh says what it holds exactly): the tensor cores multiply E2M1 weights by E4M3 terms, the TMA
// spreading the packed weights over twice their bytes as it writes them.  What bounds it: that write, 4.2 clocks a row of 64 packed bytes
// and SM, i.e. 4.4 TB/s of weights (7.0 as stored; boxes of 64 bytes as stored are as slow), and from some 80 tokens an expert on the MMAs,
// half as fast as FP4 ones.  moe_gemm_kernel.cuh, which dequantises into tensor memory, waits for its handshakes: 256 experts of 4096, 2048,
// top 6, us a layer there -> here: 2 tokens 112 -> 80, 64 tokens (Zipf) 482 -> 368, 300 tokens 924 -> 719, 1 003 tokens 995 -> 846, 2 048
// tokens 1 160 -> 1 075, 3 300 tokens 1 379 -> 1 345 (from 1 003 on at the power limit: up to 15 % more on other boxes); 32 experts of 2048,
// 1024, top 4, 300 tokens 87 -> 66.
struct MoeQFp4 {                                     // kind::mxf4: activations as three MXFP4 terms
    static constexpr int kKBlock = 256;              // K-elements per stage
    static constexpr uint32_t kBoxBytes = 128 * 128; // bytes that a box of 128 weight rows brings in
    static constexpr int kAtoms128 = 2;              // pieces of 128 K-elements (scale atoms of an operand's 128 rows) per stage
    static constexpr bool kWide = false;             // few tokens: the three terms side by side along N
};
struct MoeQFp8 {                                     // kind::mxf8f6f4: activations as three E4M3 terms, weights E2M1 in 16-byte groups
    static constexpr int kKBlock = 128;              // of 16 (8 bytes, 8 bytes of padding), which is how the TMA lays them down
    static constexpr uint32_t kBoxBytes = 128 * 64;
    static constexpr int kAtoms128 = 1;
    static constexpr bool kWide = true;
};
constexpr int kQTerms = 3;                           // activation terms
constexpr int kQTok = 112;                           // tokens per tile at most
constexpr uint32_t kQTile = 128 * 128;               // bytes of one packed weight tile (128 rows x 128 B)
// Tiles of up to CAP tokens.  Where experts have few tokens the weights' way from HBM is what a tile waits for: five stages of 32
// tokens instead of three of 112 keep more of them on it (256 experts of 4096, 2048, top 6: 17 tokens 216 -> 209.5 us, 64 zipf 278 ->
// 270, 300 579 -> 567; below ten tokens no difference).  Taken up to kQFewTokens pairs per expert, where next to no expert has more
// than 32.
constexpr int kQFewTokens = 16;
// E4M3 terms.  Us a layer, tiles of 32 tokens (terms side by side) / of 112 / dequantising (moe_gemm_kernel.cuh), one box, by pairs per expert:
//   256 experts of 4096, 2048, top 6, uniform: 8 727 / 780 / 933,  16 805 / 850 / 1 005,  20 821 / 876 / 1 031,  24 917 / 915 / 1 052,
//     28 1 025 / 936 / 1 104,  64 - / 1 180 / 1 390,  79 - / 1 490 / 1 573,  90 - / 1 690 / 1 650,  100 - / 1 755 / 1 758
//   the same, Zipf(1.1): 8 720 / 870 / 910,  12 850 / 832 / 1 003,  16 958 / 892 / 1 096,  20 1 046 / 948 / 1 156,  24 1 140 / 986 / 1 216,
//     64 - / 1 460 / 1 575,  79 - / 1 805 / 1 824,  100 - / 2 010 / 2 060
//   32 experts, top 2, uniform: 24 148 / 153 / 185,  28 164 / 156 / 186,  79 - / 198 / 241,  100 - / 229 / 262;  Zipf: 12 136 / 158 / 173,
//     24 157 / 155 / 179,  79 - / 218 / 252,  100 - / 262 / 266
// The line at 24 is where uniform routing changes over; under Zipf, whose busy experts take several tiles of 32, it is at 10, and tiles of 112
// are 5 to 13 % faster from there to 24.  The line at 80 is where dequantising is as fast for the largest bank.
constexpr int kQFewTokensFp8 = 24, kQMostTokensFp8 = 80;
constexpr int kQEpiWarps = 12, kQScaleWarps = 8;
constexpr int kQEpiGroups = kQEpiWarps / 4;          // warps per lane quadrant of tensor memory
template <class F, int CAP>
struct MoeQShape {
    static constexpr int kStages = CAP <= 32 ? 5 : 3;
    static constexpr bool kWide = F::kWide && CAP <= 32;                     // the terms side by side along N
    static constexpr int kAtoms = kWide ? 1 : kQTerms;                       // scale atoms of B per 128 K-elements
    static constexpr uint32_t kMatCols = kQTok, kAccCols = 2 * kMatCols;     // accumulator columns of a matrix; of a set
    static_assert((kWide ? kQTerms * CAP : CAP) <= kQTok, "accumulator columns");
    static constexpr uint32_t kSfCol = 2 * kAccCols;                         // scale columns: A [mat][piece] x 4, B [piece][term] x 4
    static constexpr uint32_t kBStage = kQTerms * (CAP / 2) * 128;           // activation rows of one stage and CTA
    static constexpr int kPieces = F::kAtoms128;
    static constexpr uint32_t kSfB = 2 * kPieces * 512, kSfStage = kSfB + kPieces * kAtoms * 512;      // scale atoms: [mat][piece], [piece][term]
    static constexpr int kEpiRounds = (CAP + 16 * kQEpiGroups - 1) / (16 * kQEpiGroups);
    static constexpr uint32_t kOffB = kStages * 2 * kQTile, kOffSf = kOffB + kStages * kBStage, kOffTables = kOffSf + kStages * kSfStage;
    static_assert(kSfCol + 16 + 8 * kAtoms <= 512, "tensor memory overflow");
    // dynamic shared memory: stages, then the tile and offset tables of the experts
    static __host__ __device__ __forceinline__ uint32_t smem(int n_experts) { return kOffTables + 8 * (uint32_t)(n_experts + 1) + 1024; }
    static_assert(kOffTables + 8 * (kMoeMaxExperts + 1) + 1024 + 1024 <= 227 * 1024, "shared memory overflow");
};
constexpr int kQMmaWarp = 0, kQProducerWarp = 1, kQEpiWarp = 4, kQScaleWarp = kQEpiWarp + kQEpiWarps;    // warps 2, 3: idle
constexpr int kQThreads = (kQScaleWarp + kQScaleWarps) * 32;

struct MoeQGemmArgs {
    const uint8_t* wa_s; const uint8_t* wb_s;        // E8M0 scales: up W1, W3; down W2 (wb unused)
    int rows, K, n_experts;
    const uint8_t* act_s;                            // [3][P][K / 32]
    const int* row_exp;                              // E4M3 terms: [P], exponent taken out of a slot's x (moe_act_fp8_kernel)
    long long n_pairs;
    MoeGroups g;
    uint8_t* mid_q; uint8_t* mid_s;                  // up output [3][P][rows / 2] (MXFP4) or [3][P][rows] (E4M3), [3][P][rows / 32]
    float* y;                                        // down output [P, rows] FP32
};
// Weight boxes of 128 rows; activation boxes of 3 terms x half a tile's columns, one per column count.
struct MoeQMaps { CUtensorMap wa, wb, act[kMoeWidths]; };

// What a tile is: expert, tokens, and the first weight row of the pair's first block; the same in both CTAs.
struct MoeQTile { int e, slot0, n_valid, width, m0, mats; };
constexpr int kQRows = 2 * kMoeTileRows;             // weight rows of one block of a pair
constexpr int kQTileRowsUp = kQRows, kQTileRowsDown = 2 * kQRows;

template <int MODE, int CAP>
__device__ __forceinline__ MoeQTile moe_qtile_decode(const int* tiles, const int* offsets, int n_experts, int m_tiles,
                                                     int rows, int tile) {
    int lo = 0, hi = n_experts;                      // last expert with tiles[e] <= tile
    while (hi - lo > 1) {
        const int md = (lo + hi) >> 1;
        if (tiles[md] <= tile) lo = md; else hi = md;
    }
    MoeQTile t;
    t.e = lo;
    const int local = tile - tiles[lo], nt = local / m_tiles;
    const int per = moe_tokens_per_tile(offsets[lo + 1] - offsets[lo], CAP);
    t.slot0 = offsets[lo] + nt * per;
    t.n_valid = min(per, offsets[lo + 1] - t.slot0);
    t.width = moe_width_index(t.n_valid);
    t.m0 = (local - nt * m_tiles) * (MODE == 0 ? kQTileRowsUp : kQTileRowsDown);
    t.mats = (MODE == 1 && t.m0 + kQRows >= rows) ? 1 : 2;             // a last, half down tile
    return t;
}

// A position in a ring of stages: slot and the number of times it has been filled before.
struct RingPos {
    uint32_t slot = 0, round = 0;
    __device__ __forceinline__ void next(uint32_t n) { if (++slot == n) { slot = 0; ++round; } }
};

// TMA loads of a CTA of a pair, into its own shared memory, counted on a barrier that may be the other CTA's (no
// multicast).
__device__ __forceinline__ void tma_pair_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_pair_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}

// The MMAs of one stage, by one thread, as straight-line code: a branch or a descriptor put together between two of them
// costs about 30 clocks, half of what the MMA itself takes.  The scale columns are the same in every stage: scale
// copies and MMAs of one thread execute in the order they are issued.
struct MoeQStage {
    uint64_t w, b;                                   // descriptors of the first weight tile and of term 1
    uint32_t sf, acc, sfa, b_term, idesc[4];         // (idesc: by K-step; FP4 by its parity)
    bool fresh;                                      // first stage of a tile: overwrite the accumulators
};
template <class F, class Q, int MATS>
__device__ __forceinline__ void moe_q_issue(const MoeQStage& q) {
    constexpr bool FP8 = F::kAtoms128 == 1;
    const uint32_t sfb = q.sfa + 16;
#pragma unroll
    for (int at = 0; at < Q::kPieces; ++at) {
#pragma unroll
        for (int m = 0; m < MATS; ++m) tc05_pair_copy_scale_atom(q.sfa + (m * Q::kPieces + at) * 4, q.sf + (m * Q::kPieces + at) * 512);
#pragma unroll
        for (int i = 0; i < Q::kAtoms; ++i)
            tc05_pair_copy_scale_atom(sfb + (at * Q::kAtoms + i) * 4, q.sf + Q::kSfB + (at * Q::kAtoms + i) * 512);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)                      // K-steps of 32 bytes
#pragma unroll
        for (int m = 0; m < MATS; ++m) {
            const int at = FP8 ? 0 : j >> 1;
            const uint64_t da = q.w + m * (kQTile >> 4) + 2 * j;
            const uint32_t d = q.acc + m * Q::kMatCols, sa = q.sfa + (m * Q::kPieces + at) * 4, sb = sfb + at * Q::kAtoms * 4;
            if (Q::kWide) {
                tc05_pair_mma_mx<FP8, kAOnce>(d, da, q.b + 2 * j, q.idesc[FP8 ? j : j & 1], sa, sb, (j > 0 || !q.fresh) ? 1u : 0u);
                continue;
            }
            // the three terms multiply the same A: read once, kept in the collector
            tc05_pair_mma_mx<FP8, kAFill>(d, da, q.b + 2 * j, q.idesc[FP8 ? j : j & 1], sa, sb, (j > 0 || !q.fresh) ? 1u : 0u);
            tc05_pair_mma_mx<FP8, kAUse>(d, da, q.b + q.b_term + 2 * j, q.idesc[FP8 ? j : j & 1], sa, sb + 4, 1u);
            tc05_pair_mma_mx<FP8, kALast>(d, da, q.b + 2 * q.b_term + 2 * j, q.idesc[FP8 ? j : j & 1], sa, sb + 8, 1u);
        }
}

// Terms side by side (N = 3 x tokens): column i * half + j of CTA r's half of the columns (they start at 3 half r) is term i of token
// r * half + j, half = 8 or 16.  Both ways the 48 columns from 3 c on are those of the 16 tokens from c on: their sums.
__device__ __forceinline__ void moe_q_sum_terms(uint32_t tcol, int half, uint32_t (&p)[16]) {
    uint32_t q[kQTerms][16];
#pragma unroll
    for (int i = 0; i < kQTerms; ++i) tc05_ld16_issue(tcol + 16 * i, q[i]);
    tc05_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int w = (j >> 3) * 24 + (j & 7);
        const float a = __uint_as_float(half == 8 ? q[w >> 4][w & 15] : q[0][j]);
        const float b = __uint_as_float(half == 8 ? q[(w + 8) >> 4][(w + 8) & 15] : q[1][j]);
        const float c = __uint_as_float(half == 8 ? q[(w + 16) >> 4][(w + 16) & 15] : q[2][j]);
        p[j] = __float_as_uint((a + b) + c);
    }
}

// Tokens and lanes trade places: on entry v[i] is token i of row `lane` of a 32-row block, on return v[j] is row
// 16 (lane / 16) + j of token lane % 16 (a 16 x 16 transpose in each half of the warp, four exchange steps).
__device__ __forceinline__ void moe_transpose16(float (&v)[16], int lane) {
#pragma unroll
    for (int bit = 8; bit > 0; bit >>= 1) {
        const bool up = (lane & bit) != 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (i & bit) continue;
            const float lo = v[i], hi = v[i + bit];
            const float got = __shfl_xor_sync(kFullMask, up ? lo : hi, bit);
            v[i] = up ? got : lo;
            v[i + bit] = up ? hi : got;
        }
    }
}

// Half a 32-element block per lane (the other half in lane ^ 16) -> three MXFP4 terms: 8 packed bytes and the block's
// scale byte each.  The rule of the terms is moe_quantize_mxfp4x3's; the residual is kept in units of the last scale, so that a
// term needs no multiplication back.
__device__ __forceinline__ void moe_quantize_half_block(float (&v)[16], uint2 (&packed)[kQTerms], uint32_t (&scale)[kQTerms]) {
    int unit = 127;                                  // v is in units of 2^(unit - 127)
#pragma unroll
    for (int t = 0; t < kQTerms; ++t) {
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
        m = max(m, __shfl_xor_sync(kFullMask, m, 16));
        int e = (int)((m + 0x003fffffu) >> 23) - 2 + (unit - 127);        // biased; smallest with amax <= 6 * 2^(e - 127)
        e = min(max(e, 0), 254);
        const float inv = __uint_as_float((uint32_t)min(max(127 + unit - e, 1), 254) << 23);
        unit = e;
        scale[t] = (uint32_t)e;
        uint32_t r[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            uint16_t q;
            v[i] *= inv;
            v[i + 1] *= inv;
            asm("{\n .reg .b8 b;\n cvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n mov.b16 %0, {b, 0};\n}"
                : "=h"(q) : "f"(v[i]), "f"(v[i + 1]));
            if (t + 1 < kQTerms) {
                const float2 back = e2m1x2_to_float2(q);
                v[i] -= back.x;
                v[i + 1] -= back.y;
            }
            r[i >> 3] |= (uint32_t)(q & 0xff) << (4 * (i & 7));
        }
        packed[t] = make_uint2(r[0], r[1]);
    }
}

// The same -> three E4M3 terms (moe_quantize_e4m3x3), 16 bytes each.
__device__ __forceinline__ void moe_quantize_half_block_fp8(float (&v)[16], uint4 (&packed)[kQTerms], uint32_t (&scale)[kQTerms]) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = max(m, __float_as_uint(v[i]) & 0x7fffffffu);
    m = max(m, __shfl_xor_sync(kFullMask, m, 16));
    moe_quantize_e4m3x3<kE4m3MidStep>(v, m, packed, scale);
}

template <int MODE, int CAP, class F>
__global__ void __launch_bounds__(kQThreads, 1) moe_gemm_mxf4_kernel(const __grid_constant__ MoeQMaps maps, const MoeQGemmArgs a) {
    using Q = MoeQShape<F, CAP>;
    constexpr bool FP8 = F::kAtoms128 == 1;
    constexpr int kQStages = Q::kStages, kQEpiRounds = Q::kEpiRounds;
    constexpr uint32_t kQSfStage = Q::kSfStage;
    extern __shared__ __align__(1024) uint8_t gemm_smem[];
    __shared__ __align__(8) uint64_t full[kQStages], empty[kQStages], acc_full[2], acc_free[2];
    __shared__ uint32_t tmem_holder;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_st = a.K / F::kKBlock, row_s = a.K >> 5;
    const uint32_t smem_w = smem_u32(gemm_smem), smem_b = smem_w + Q::kOffB, smem_sf = smem_w + Q::kOffSf;
    int* const s_tiles = reinterpret_cast<int*>(gemm_smem + Q::kOffTables);
    int* const s_offsets = s_tiles + a.n_experts + 1;

    if (warp == kQMmaWarp) tc05_pair_alloc(smem_u32(&tmem_holder), 512);
    if (tid == 0) {
        for (int s = 0; s < kQStages; ++s) { mbar_init(smem_u32(&full[s]), 2 * (1 + kQScaleWarps / 2)); mbar_init(smem_u32(&empty[s]), 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&acc_full[s]), 1); mbar_init(smem_u32(&acc_free[s]), 2 * kQEpiWarps); }
        mbar_init_fence();
    }
    // The tables come from the kernel before the one this launch depends on: a grid starts its dependents only after its own
    // wait, so that kernel is complete; what the previous kernel wrote (the activations) is waited for by the roles that
    // read it, and the first weights are requested before that.
    for (int i = tid; i <= a.n_experts; i += kQThreads) {
        s_tiles[i] = __ldcg((MODE == 0 ? a.g.tiles_up : a.g.tiles_down) + i);
        s_offsets[i] = __ldcg(a.g.offsets + i);
    }
    tc05_fence_before_sync();
    cluster_sync_all();                                       // barriers of both CTAs are initialised
    tc05_fence_after_sync();
    const uint32_t tmem = tmem_holder;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    auto leader = [&](uint64_t& bar) { return cluster_map(smem_u32(&bar), 0); };
    const int n_tiles = s_tiles[a.n_experts];
    const int m_tiles = (a.rows + (MODE == 0 ? kQTileRowsUp : kQTileRowsDown) - 1) / (MODE == 0 ? kQTileRowsUp : kQTileRowsDown);
    auto decode = [&](int tile) { return moe_qtile_decode<MODE, CAP>(s_tiles, s_offsets, a.n_experts, m_tiles, a.rows, tile); };
    bool alive = true;
    auto wait = [&](uint64_t& bar, uint32_t parity, int code) {            // roles of whole warps
        if (alive) alive = __all_sync(kFullMask, mbar_wait_bounded(smem_u32(&bar), parity & 1u, code));
    };
    auto wait_one = [&](uint64_t& bar, uint32_t parity, int code) {        // roles of one thread
        if (alive) alive = mbar_wait_bounded(smem_u32(&bar), parity & 1u, code);
    };
    uint32_t tc = 0;                                          // tiles begun by this pair

    if (warp >= kQEpiWarp && warp < kQScaleWarp) {
        const int quad = warp & 3, r = quad * 32 + lane;
        pdl_wait();
        for (int tile = pair; tile < n_tiles; tile += n_pairs, ++tc) {
            const MoeQTile t = decode(tile);
            const uint32_t buf = tc & 1u;
            const int m0 = t.m0 + rank * kMoeTileRows;        // first row of this CTA in block 0
            // lanes i and i + 16 hold, for token i of each of this warp's chunks: down, the router weight; of E4M3 terms, the power of two
            // that was taken out of x and so of G and of U.  G gets it back before the sigmoid, y with the weight.
            float w[kQEpiRounds];
            if (MODE == 1 || FP8)
#pragma unroll
                for (int i = 0; i < kQEpiRounds; ++i) {
                    const int n = (((warp - kQEpiWarp) >> 2) + kQEpiGroups * i) * 16 + (lane & 15);
                    w[i] = MODE == 1 ? 0.f : 1.f;
                    if (n < t.n_valid) {
                        if (MODE == 1) w[i] = __ldcg(a.g.slot_w + t.slot0 + n);
                        if (FP8) w[i] *= float_pow2(__ldcg(a.row_exp + t.slot0 + n));
                    }
                }
            wait(acc_full[buf], tc >> 1, 6);
            tc05_fence_after_sync();
            const uint32_t trow = tmem + ((uint32_t)(quad * 32) << 16) + buf * Q::kAccCols;
            // the warps of a lane quadrant take chunks of 16 tokens in turn
#pragma unroll
            for (int k = 0; k < kQEpiRounds; ++k) {
                const int c = (((warp - kQEpiWarp) >> 2) + kQEpiGroups * k) * 16;
                if (c >= t.n_valid || !alive) break;
                const int n = min(16, t.n_valid - c);
                auto sums = [&](int m, uint32_t (&p)[16]) {   // of block m; wide: complete on return
                    if constexpr (Q::kWide) moe_q_sum_terms(trow + m * Q::kMatCols + 3 * c, moe_width(t.width, CAP) >> 1, p);
                    else tc05_ld16_issue(trow + m * Q::kMatCols + c, p);
                };
                uint32_t p0[16], p1[16];
                sums(0, p0);
                if (MODE == 0 || !Q::kWide) sums(1, p1);      // (stale, and not used, in a half tile)
                if (!Q::kWide) tc05_wait_ld();
                if (MODE == 0) {
                    float g[16];
                    if (FP8 && __any_sync(kFullMask, w[k] != 1.f)) {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            p0[i] = __float_as_uint(saturate_finite(__uint_as_float(p0[i]) * __shfl_sync(kFullMask, w[k], i)));
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float gate = __uint_as_float(p0[i]);
                        const float v = __fdividef(gate, 1.0f + __expf(-gate)) * __uint_as_float(p1[i]);
                        g[i] = i < n ? (FP8 ? saturate_finite(v) : v) : 0.f;
                    }
                    moe_transpose16(g, lane);
                    typename std::conditional<FP8, uint4, uint2>::type packed[kQTerms];
                    uint32_t scale[kQTerms];
                    if constexpr (FP8) moe_quantize_half_block_fp8(g, packed, scale);
                    else moe_quantize_half_block(g, packed, scale);
                    const int i = lane & 15;
                    const long long slot = t.slot0 + c + i;
                    if (i < n) {
                        const int h0 = m0 + quad * 32;
#pragma unroll
                        for (int q = 0; q < kQTerms; ++q) {
                            const long long at = (q * a.n_pairs + slot) * a.rows + h0;          // element
                            if constexpr (FP8) *reinterpret_cast<uint4*>(a.mid_q + at + (lane >> 4) * 16) = packed[q];
                            else *reinterpret_cast<uint2*>(a.mid_q + (at >> 1) + (lane >> 4) * 8) = packed[q];
                            if (lane < 16) a.mid_s[(q * a.n_pairs + slot) * (a.rows >> 5) + (h0 >> 5)] = (uint8_t)scale[q];
                        }
                    }
                } else {
                    auto put = [&](const uint32_t (&p)[16], int row) {
                        if (row >= a.rows) return;                                                        // (a.rows is a multiple of 128)
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float wi = __shfl_sync(kFullMask, w[k], i);
                            if (i < n) a.y[(size_t)(t.slot0 + c + i) * a.rows + row + r] = __uint_as_float(p[i]) * wi;
                        }
                    };
                    put(p0, m0);
                    if (Q::kWide && t.mats == 2) sums(1, p1);
                    put(p1, m0 + kQRows);
                }
            }
            tc05_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader(acc_free[buf]));
        }
    } else if (warp >= kQScaleWarp) {
        // ---- scale bytes: a word per row and 128 K-elements.  Thread st of a group holds weight row st of both matrices and token st of
        // every term.  A load, 16 bytes of a row or 8, is a run of kRun stages; a group takes every second run, and its next run is loaded
        // before the current one is stored, whichever tile it belongs to.  Between a group's runs lies one of the other's: only with more
        // stages in the ring than kRun has it seen the slot's last but one use end, without which a parity says nothing.
        constexpr int kRun = 4 / Q::kPieces < kQStages ? 4 / Q::kPieces : 2;
        static_assert(kQStages > kRun, "a scale group may not run ahead of a slot by two phases");
        const int st = (tid - kQScaleWarp * 32) & 127, group = (warp - kQScaleWarp) >> 2;
        const int n_prs = (n_st + kRun - 1) / kRun;
        int tile = pair, count = 0, pr = group;               // next run to load: pr of tile number `count`
        const uint8_t* src[2 + kQTerms] = {};
        bool fresh = true;
        struct Loaded { uint4 v[2 + kQTerms]; uint32_t has; uint32_t it; int stages, half; };
        int half = 0;                                          // token columns of a CTA
        auto load = [&](Loaded& l) -> bool {
            while (pr >= n_prs) { pr -= n_prs; tile += n_pairs; ++count; fresh = true; }
            if (tile >= n_tiles) return false;
            if (fresh) {
                const MoeQTile t = decode(tile);
                const int m0 = t.m0 + rank * kMoeTileRows;
                const long long first = (long long)t.e * a.rows + m0 + st;
                src[0] = m0 < a.rows ? a.wa_s + first * row_s : nullptr;
                src[1] = MODE == 0 ? a.wb_s + first * row_s : m0 + kQRows < a.rows ? a.wa_s + (first + kQRows) * row_s : nullptr;
#pragma unroll
                for (int i = 0; i < kQTerms; ++i)
                    src[2 + i] = st < t.n_valid ? a.act_s + (i * a.n_pairs + t.slot0 + st) * row_s : nullptr;
                half = moe_width(t.width, CAP) >> 1;
                fresh = false;
            }
            l.half = half;
            l.has = 0;
            l.it = (uint32_t)count * n_st + kRun * pr;
            l.stages = min(kRun, n_st - kRun * pr);
#pragma unroll
            for (int i = 0; i < 2 + kQTerms; ++i) {
                if (!src[i]) continue;
                l.has |= 1u << i;
                if (kRun * Q::kPieces == 2) {
                    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(src[i]) + pr);
                    l.v[i] = make_uint4(v.x, v.y, 0, 0);
                } else if ((row_s & 15) == 0) {                // otherwise the rows are 8-byte aligned
                    l.v[i] = __ldcg(reinterpret_cast<const uint4*>(src[i]) + pr);
                } else {
                    const uint2* p = reinterpret_cast<const uint2*>(src[i]) + 2 * pr;
                    const uint2 lo = __ldcg(p), hi = l.stages == kRun ? __ldcg(p + 1) : make_uint2(0, 0);
                    l.v[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
                }
            }
            pr += 2;
            return true;
        };
        const uint32_t atom = tc05_scale_atom_offset(st, 0);
        // Stage n of a run.  (Written as a loop over the run, unrolled, this role held up the gate/up GEMM of few tokens: 64 tokens 280 ->
        // 302 us, 600 tokens 374 -> 406.)
        auto put_stage = [&](const Loaded& l, uint32_t it, int n) {
            const uint32_t slot = it % kQStages, round = it / kQStages;
            if (round > 0) wait(empty[slot], round - 1, 4);
            const uint32_t sf = smem_sf + slot * kQSfStage;
#pragma unroll
            for (int i = 0; i < 2 + kQTerms; ++i)
                if (l.has & (1u << i)) {
                    uint32_t at = sf + atom + (i < 2 ? i * Q::kPieces * 512u : Q::kSfB + (i - 2) * 512u);
                    if (Q::kWide && i >= 2)                    // a column per term and token: see moe_q_sum_terms
                        at = sf + Q::kSfB + tc05_scale_atom_offset(st + (i - 2 + (st >= l.half ? kQTerms - 1 : 0)) * l.half, 0);
                    const uint4& v = l.v[i];
                    if (FP8) {                                 // one piece of 128 K-elements, or two
                        uint32_t word = n == 0 ? v.x : n == 1 ? v.y : n == 2 ? v.z : v.w;
                        if (i < 2) word &= ~__vcmpeq4(word, 0xffffffffu);      // a weight's 0xFF contributes nothing on this path: 2^-127
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(word) : "memory");
                    } else {
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(n == 1 ? v.z : v.x) : "memory");
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + (i < 2 ? 512u : Q::kAtoms * 512u)), "r"(n == 1 ? v.w : v.y) : "memory");
                    }
                }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader(full[slot]));
        };
        auto put = [&](const Loaded& l) {
            put_stage(l, l.it, 0);
            if (l.stages > 1) put_stage(l, l.it + 1, 1);
            if (kRun == 4 && l.stages > 2) {                   // (an even number of stages a tile)
                put_stage(l, l.it + 2, 2);
                put_stage(l, l.it + 3, 3);
            }
        };
        pdl_wait();
        Loaded l0, l1;
        bool more = load(l0);
        while (more) {
            more = load(l1);
            put(l0);
            if (!more) break;
            more = load(l0);
            put(l1);
        }
    } else if (warp == kQProducerWarp) {
        // ---- this role and the MMAs are one thread each: nothing in their loops is done by a warp, so no vote or
        // reconvergence stands between a barrier and what follows it
        if (tc05_elect_one()) {
            RingPos pos;
            bool waited = false;
            MoeQTile t = {}, next = {};                       // the next tile is looked up while this one's stages are on their way
            if (pair < n_tiles) t = decode(pair);
            for (int tile = pair; tile < n_tiles && alive; tile += n_pairs, t = next) {
                const int first = t.e * a.rows + t.m0 + rank * kMoeTileRows;      // past the expert in a half tile: loaded, not used
                const int half = moe_width(t.width, CAP) >> 1, slot = t.slot0 + rank * half;
                const CUtensorMap* act = &maps.act[t.width];
                const uint32_t bytes = t.mats * F::kBoxBytes + kQTerms * half * 128u;
                auto weights = [&](int s, const RingPos& p) {
                    const uint32_t bar = leader(full[p.slot]), dst = smem_w + p.slot * 2 * kQTile;
                    mbar_arrive_expect_tx_cluster(bar, bytes);
                    tma_pair_load_2d(dst, &maps.wa, s * 128, first, bar);
                    if (t.mats == 2) tma_pair_load_2d(dst + kQTile, &maps.wb, s * 128, first + (MODE == 0 ? 0 : kQRows), bar);
                };
                auto tokens = [&](int s, const RingPos& p) {
                    tma_pair_load_3d(smem_b + p.slot * Q::kBStage, act, s * 128, slot, 0, leader(full[p.slot]));
                };
                int s0 = 0;
                if (!waited) {                                // the pair's first stages: weights before the wait
                    s0 = min(n_st, kQStages);
                    RingPos p;
                    for (int s = 0; s < s0; ++s, p.next(kQStages)) weights(s, p);
                    pdl_wait();
                    pdl_launch_dependents();                  // after the wait: the next kernel reads the tile tables before its own
                    waited = true;
                    for (int s = 0; s < s0; ++s, pos.next(kQStages)) tokens(s, pos);
                }
                for (int s = s0; s < n_st; ++s, pos.next(kQStages)) {
                    if (pos.round > 0) wait_one(empty[pos.slot], pos.round - 1, 4);
                    if (!alive) break;
                    weights(s, pos);
                    tokens(s, pos);
                    if (s == n_st >> 1 && tile + n_pairs < n_tiles) next = decode(tile + n_pairs);
                }
                if (s0 > n_st >> 1 && tile + n_pairs < n_tiles) next = decode(tile + n_pairs);
            }
            if (!waited) { pdl_wait(); pdl_launch_dependents(); }
        }
        __syncwarp();
    } else if (warp == kQMmaWarp) {
        if (rank == 0 && tc05_elect_one()) {
            RingPos pos;
            MoeQTile t = {}, next = {};
            if (pair < n_tiles) t = decode(pair);
            for (int tile = pair; tile < n_tiles && alive; tile += n_pairs, ++tc, t = next) {
                const uint32_t buf = tc & 1u;
                const int n = moe_width(t.width, CAP);
                MoeQStage q;
                q.acc = tmem + buf * Q::kAccCols;
                q.sfa = tmem + Q::kSfCol;
                q.b_term = (uint32_t)n * 4;                   // 128 n / 2 bytes, in the descriptor's units
#pragma unroll
                for (int j = 0; j < (FP8 ? 4 : 2); ++j) {     // scale bytes of K-step j: two of every four, or one
                    const int id = FP8 ? j : 2 * j;
                    const int cols = Q::kWide ? kQTerms * n : n;
                    q.idesc[j] = FP8 ? tc05_idesc_mxf8f6f4(256, cols, id, id) : tc05_idesc_mxf4(256, cols, id, id);
                }
                if (tc >= 2) wait_one(acc_free[buf], (tc >> 1) - 1, 7);
                for (int s = 0; s < n_st; ++s, pos.next(kQStages)) {
                    wait_one(full[pos.slot], pos.round, 5);
                    if (!alive) break;
                    tc05_fence_after_sync();
                    q.w = tc05_desc_k_sw128(smem_w + pos.slot * 2 * kQTile);
                    q.b = tc05_desc_k_sw128(smem_b + pos.slot * Q::kBStage);
                    q.sf = smem_sf + pos.slot * kQSfStage;
                    q.fresh = s == 0;
                    if (t.mats == 2) moe_q_issue<F, Q, 2>(q); else moe_q_issue<F, Q, 1>(q);
                    tc05_pair_commit(smem_u32(&empty[pos.slot]));
                    if (s == n_st >> 1 && tile + n_pairs < n_tiles) next = decode(tile + n_pairs);
                    if (s == n_st - 1) tc05_pair_commit(smem_u32(&acc_full[buf]));
                }
            }
        }
        __syncwarp();
    }
    tc05_fence_before_sync();
    cluster_sync_all();                                       // no arrival for this CTA is still on its way
    tc05_fence_after_sync();
    if (warp == kQMmaWarp) tc05_pair_dealloc(tmem, 512);
}

}  // namespace dsv4
