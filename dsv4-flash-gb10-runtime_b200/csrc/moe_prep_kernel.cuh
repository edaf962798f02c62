// Preparation of the batched layer, two launches: the pairs grouped by expert, then the activations in the form the
// tensor-core path wants - three MXFP4 or E4M3 terms, or normalised fp16 - written once per PAIR in slot order, so that the rows
// of a tile are neighbours and the GEMM fetches them with one copy per stage instead of one gather per four rows.
#pragma once

#include "moe_prep.cuh"
#include "stream_ring.cuh"

namespace dsv4 {

constexpr int kPrepThreads = 1024;
// Grouping: one block up to this many pairs, a cluster of eight above (24 576 pairs took a single block 26 us).
constexpr int kGroupOneBlockPairs = 2048;
constexpr int kGroupCluster = 8;

constexpr int kTypicalRows = 16;                           // weight rows looked at per expert and matrix
constexpr int kTypicalExperts = kPrepThreads / 32 / 4;     // experts of a block: four warps each

// The typical scale byte of W1 and of W3 of a few experts, by a block: the mean E8M0 byte of some of their rows (bytes 0 and 255, i.e.
// zero blocks and NaN, left out).  It only centres the range of the intermediate; any value near the truth will do.  A warp takes half of
// an expert's rows of one matrix.  (A warp for a whole expert, its bytes counted one by one, made the launch 12 us longer.)
struct MoeTypicalArgs {
    const uint8_t* w1_s; const uint8_t* w3_s;              // E8M0 bytes [E, hidden, K / 32]
    int K, hidden, n_experts;
    int* typical;                                          // [E] out: typical byte of W1 | of W3 << 8
};
__device__ __forceinline__ void moe_typical_scales(const MoeTypicalArgs& a, int block) {
    __shared__ int part[kPrepThreads / 32][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = block * kTypicalExperts + (warp >> 2);
    const int row_s = a.K >> 5, words = row_s >> 2, step = max(1, a.hidden / kTypicalRows);
    int sum = 0, n = 0;
    if (e < a.n_experts) {
        const uint8_t* base = (warp & 2 ? a.w3_s : a.w1_s) + (long long)e * a.hidden * row_s;
        const int r0 = (warp & 1) * (kTypicalRows / 2);
        for (int c = lane; c < words; c += 32) {
            uint32_t w[kTypicalRows / 2];
#pragma unroll
            for (int i = 0; i < kTypicalRows / 2; ++i)
                w[i] = __ldg(reinterpret_cast<const uint32_t*>(base + (long long)min((r0 + i) * step, a.hidden - 1) * row_s) + c);
#pragma unroll
            for (int i = 0; i < kTypicalRows / 2; ++i) {
                const uint32_t f = w[i] & ~__vcmpeq4(w[i], 0xffffffffu);           // 0xFF and 0 add nothing
                sum = __dp4a(f, 0x01010101u, (uint32_t)sum);
                n += __popc((((f & 0x7f7f7f7fu) + 0x7f7f7f7fu) | f) & 0x80808080u);
            }
        }
    }
    sum = __reduce_add_sync(kFullMask, sum);
    n = __reduce_add_sync(kFullMask, n);
    if (lane == 0) { part[warp][0] = sum; part[warp][1] = n; }
    __syncthreads();
    if (threadIdx.x >= kTypicalExperts || block * kTypicalExperts + (int)threadIdx.x >= a.n_experts) return;
    int typ[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int* p = part[4 * threadIdx.x + 2 * m];
        const int s = p[0] + p[2], c = p[1] + p[3];
        typ[m] = c > 0 ? (s + c / 2) / c : 127;
    }
    a.typical[block * kTypicalExperts + threadIdx.x] = typ[0] | (typ[1] << 8);
}

struct MoeGroupArgs {
    const int* ids;                  // [P] expert of every pair, negative = skip
    const float* weights;            // [P]
    int n_pairs, n_experts, m_tiles_up, m_tiles_down, tile_tokens;
    int blocks;                      // that sort; where the grid has more, they look for the typical scales
    MoeTypicalArgs typical;
    MoeGroups g;
    int* status;
};

// Counting sort of the pairs by expert.  The order of pairs inside an expert is arbitrary (it only decides which
// accumulator column a token uses, not any arithmetic).  Every block of the cluster takes a contiguous part of the pairs;
// the blocks read one another's counts.  Thread e owns expert e (kPrepThreads == kMoeMaxExperts).
__global__ void __launch_bounds__(kPrepThreads) moe_group_kernel(const MoeGroupArgs a) {
    __shared__ int count[kMoeMaxExperts], cursor[kMoeMaxExperts], warp_sums[2][32];
    pdl_wait();
    pdl_launch_dependents();                               // after the wait: the next kernel reads x before its own
    const int e = threadIdx.x, lane = e & 31, wid = e >> 5;
    const int blocks = a.blocks, blk = blockIdx.x;
    if (blk >= blocks) {                                   // (whole clusters of them)
        moe_typical_scales(a.typical, blk - blocks);
        return;
    }
    count[e] = 0;
    __syncthreads();
    const int per = (a.n_pairs + blocks - 1) / blocks;
    const int p0 = min(a.n_pairs, blk * per), p1 = min(a.n_pairs, p0 + per);
    constexpr int kBatch = 4;                              // independent loads in flight per thread
    for (int b = p0 + e; b < p1; b += kPrepThreads * kBatch) {
        int id[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) id[i] = b + i * kPrepThreads < p1 ? __ldcg(a.ids + b + i * kPrepThreads) : -1;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            if (id[i] >= a.n_experts) atomicExch(a.status, 3);     // past the bank: dropped and reported
            else if (id[i] >= 0) atomicAdd(&count[id[i]], 1);      // negative: another rank's expert, dropped silently
        }
    }
    int total = 0, before = 0;
    if (blocks == 1) {
        __syncthreads();
        total = count[e];
    } else {
        cluster_sync_all();
        for (int r = 0; r < blocks; ++r) {
            int c;
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(c) : "r"(cluster_map(smem_u32(&count[e]), r)));
            before += r < blk ? c : 0;
            total += c;
        }
        cluster_sync_all();                                // everyone has read the counts: a block may leave
    }
    // exclusive prefix sums over the experts of pairs and of token tiles
    const int v[2] = {total, moe_token_tiles(total, a.tile_tokens)};
    int inc[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        int x = v[q];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(kFullMask, x, off);
            if (lane >= off) x += y;
        }
        inc[q] = x;
        if (lane == 31) warp_sums[q][wid] = x;
    }
    __syncthreads();
    if (wid < 2) {
        int x = warp_sums[wid][lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(kFullMask, x, off);
            if (lane >= off) x += y;
        }
        warp_sums[wid][lane] = x;
    }
    __syncthreads();
    int exc[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) exc[q] = inc[q] - v[q] + (wid > 0 ? warp_sums[q][wid - 1] : 0);
    if (blk == 0 && e < a.n_experts) {
        a.g.offsets[e] = exc[0];
        a.g.tiles_up[e] = exc[1] * a.m_tiles_up;
        a.g.tiles_down[e] = exc[1] * a.m_tiles_down;
        if (e == a.n_experts - 1) {
            a.g.offsets[a.n_experts] = exc[0] + v[0];
            a.g.tiles_up[a.n_experts] = (exc[1] + v[1]) * a.m_tiles_up;
            a.g.tiles_down[a.n_experts] = (exc[1] + v[1]) * a.m_tiles_down;
        }
    }
    cursor[e] = exc[0] + before;
    __syncthreads();
    for (int b = p0 + e; b < p1; b += kPrepThreads * kBatch) {
        int id[kBatch];
        float w[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int p = b + i * kPrepThreads;
            id[i] = p < p1 ? __ldcg(a.ids + p) : -1;
            w[i] = p < p1 ? __ldcg(a.weights + p) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int p = b + i * kPrepThreads;
            if (p >= p1) continue;
            int slot = -1;
            if (id[i] >= 0 && id[i] < a.n_experts) {
                slot = atomicAdd(&cursor[id[i]], 1);
                a.g.slot_w[slot] = w[i];
            }
            a.g.pair_slot[p] = slot;
        }
    }
}

struct MoeActArgs {
    const __nv_bfloat16* x;          // [T, K] (peer form: rows come from the ranks that published them)
    const int* pair_slot;            // [T, k]
    int n_tokens, k, K;
    long long n_pairs;
    uint8_t* q; uint8_t* s;          // block-scaled MMAs, out: terms [3][P][K / 2] (MXFP4) or [3][P][K] (E4M3), scales [3][P][K / 32]
    __half* xh;                      // fp16 MMAs, out: [P, K]
    int2* xexp;                      // fp16 MMAs, [P] out: {exponent removed from x, floor(log2(rms of what is left))}
    const int* ids;                  // E4M3 terms: [T, k]
    int* row_exp;                    // E4M3 terms, [P] out: exponent removed from x
    MoeTypicalArgs typical;          // fp16 MMAs: the first blocks write them; E4M3 terms: read
};

template <bool PEER>
__device__ __forceinline__ const __nv_bfloat16* moe_act_row(const MoeActArgs& a, const MoePeerIn& in, int row) {
    if (!PEER) return a.x + (long long)row * a.K;
    const int r = row / in.tokens_per_rank;
    return in.x[r] + (long long)(row - r * in.tokens_per_rank) * a.K;
}
// A token none of whose pairs has a slot is not needed (expert parallel: all its experts are on other ranks).
__device__ __forceinline__ bool moe_act_wanted(const MoeActArgs& a, int row) {
    bool wanted = false;
    for (int j = 0; j < a.k; ++j) wanted |= __ldcg(a.pair_slot + (long long)row * a.k + j) >= 0;
    return wanted;
}

// Three MXFP4 terms.  A warp takes 256 neighbouring elements of a row (K is a multiple of 256), the lanes eight each; the
// next piece and the slots of its row are on their way while this one is quantised (reading the slots one after another
// where they are used made this kernel wait for k L2 round trips per piece: 333 us for 16 384 tokens).  The rows are input of the
// layer, complete before the grouping kernel started, so the first piece is read before waiting for the slots.
template <bool PEER>
__global__ void __launch_bounds__(256, 6) moe_act_mxf4_kernel(const MoeActArgs a, const MoePeerIn in) {
    const int lane = threadIdx.x & 31;
    const int per_row = a.K >> 8, warps = gridDim.x * (blockDim.x >> 5);
    const int n_chunks = a.n_tokens * per_row;
    const long long term_q = a.n_pairs * (a.K >> 1), term_s = a.n_pairs * (a.K >> 5);
    auto slots_of = [&](int w) -> int {                        // lane j: slot of the j-th pair of the piece's token
        return w < n_chunks && lane < a.k ? __ldcg(a.pair_slot + (long long)(w / per_row) * a.k + lane) : -1;
    };
    auto fetch = [&](int w, uint4& u) {
        const int row = w / per_row;
        if (w < n_chunks && (!PEER || moe_act_wanted(a, row)))
            u = __ldcs(reinterpret_cast<const uint4*>(moe_act_row<PEER>(a, in, row) + (w - row * per_row) * 256) + lane);
    };
    if (PEER) pdl_wait();
    uint4 cur = make_uint4(0, 0, 0, 0), nxt = cur;
    int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    fetch(w, cur);
    if (!PEER) pdl_wait();
    pdl_launch_dependents();                               // after the wait: the next kernel reads the tile tables before its own
    int slots = slots_of(w);
    for (; w < n_chunks; w += warps) {
        fetch(w + warps, nxt);
        const int next_slots = slots_of(w + warps);
        const uint32_t u[4] = {cur.x, cur.y, cur.z, cur.w};
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(u[i] << 16);
            v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
        uint32_t word[3], scale[3];
        moe_quantize_mxfp4x3(v, word, scale);
        // lane 8 t + b (t < 3): scale byte b of term t
        uint32_t sb = __shfl_sync(kFullMask, scale[0], 4 * (lane & 7));
        const uint32_t sb1 = __shfl_sync(kFullMask, scale[1], 4 * (lane & 7)), sb2 = __shfl_sync(kFullMask, scale[2], 4 * (lane & 7));
        if (lane >= 8) sb = lane >= 16 ? sb2 : sb1;
        const int row = w / per_row, c = w - row * per_row;
        for (int j = 0; j < a.k; ++j) {
            const int slot = j < 32 ? __shfl_sync(kFullMask, slots, j) : __ldcg(a.pair_slot + (long long)row * a.k + j);
            if (slot < 0) continue;
            uint8_t* q = a.q + (long long)slot * (a.K >> 1) + c * 128 + 4 * lane;
#pragma unroll
            for (int t = 0; t < 3; ++t) *reinterpret_cast<uint32_t*>(q + t * term_q) = word[t];
            if (lane < 24) a.s[(lane >> 3) * term_s + (long long)slot * (a.K >> 5) + c * 8 + (lane & 7)] = (uint8_t)sb;
        }
        cur = nxt;
        slots = next_slots;
    }
}

// The same for many tokens: a lane takes a whole block of 32 elements, a warp 1024 of a row.  The form above spends the time on its
// stores (four bytes per lane, term and pair) and on the maxima of a block, two shuffles per term; here a term of a pair is one 16-byte
// store per lane and a block has no shuffles.  2 K bytes of a token come in, 51 K / 32 of each of its pairs go out.  Measured at K 4096, six
// pairs a token, the form above -> this one: 4 096 tokens 55 -> 42 us, 16 384 tokens 195 -> 155 (0.64 GB out, 0.13 in: 5.0 TB/s, three
// quarters of the copy rate; what holds the rest back has not been looked at).
// When it is taken: a quarter of the warps, each with four times the work, has to fill the SMs, and a row that is no multiple of 1024 long
// leaves lanes of its last warp idle.  Us of the stage, form above / this one (the same kernel differs by up to 0.9 between runs below 10):
//   K 4096: 128 tokens 8.2-9.0 / 9.0,  256 10.2 / 8.2-9.1,  512 12.3-13.2 / 10.2-11.2;   K 7168: 256 12.3 / 10.2
//   K 2048: 256 8.9 / 8.2-9.1, 512 10.2 / 8.2-9.0;   K 1024: 256 8.2 / 8.2-9.2, 512 8.2-9.1 / 8.2-9.1, 1 024 9.3-10.2 / 8.4-9.1, 4 096 18.5 / 15.0
//   K 2304: 512 10.2 / 10.4, 1 024 13.3 / 12.3-13.2, 4 096 33.7 / 27.4;   K 2816: 512 10.3 / 11.0, 1 024 14.4-15.3 / 12.4-13.1
//   K 1280: 1 024 10.3 / 10.2, 4 096 22.5 / 19.6;   K 768: 1 024 8.2 / 8.4, 4 096 16.4 / 14.3
//   K 512: 4 096 12.7 / 13.1;   K 256: 256 7.2 / 9.2, 4 096 9.7 / 12.6, 16 384 18.4 / 29.1
__host__ __forceinline__ bool moe_act_by_blocks(int n_tokens, int K) {
    if ((K & 1023) == 0) return n_tokens >= 256 && (long long)n_tokens * (K >> 10) >= 1024;
    return K > 1024 ? n_tokens >= 1024 : K > 512 && n_tokens >= 4096;
}

// The same bytes as above.  Rows of this GPU only: a form that kept four loads of a row in flight over NVLink disagreed once, on eight
// GPUs, and the cause is not known; rows of other ranks stay with the form above, whose runs on several GPUs agreed.
__global__ void __launch_bounds__(256, 2) moe_act_blocks_kernel(const MoeActArgs a) {
    const int lane = threadIdx.x & 31;
    const int per_row = (a.K + 1023) >> 10, warps = gridDim.x * (blockDim.x >> 5), n_pieces = a.n_tokens * per_row;
    const long long term_q = a.n_pairs * (a.K >> 1), term_s = a.n_pairs * (a.K >> 5);
    auto slots_of = [&](int w) -> int {                        // lane j: slot of the j-th pair of the piece's token
        return w < n_pieces && lane < a.k ? __ldcg(a.pair_slot + (long long)(w / per_row) * a.k + lane) : -1;
    };
    auto fetch = [&](int w, uint4 (&u)[4]) {
        const int row = w / per_row, at = (w - row * per_row) * 1024 + lane * 32;
        if (w < n_pieces && at < a.K) {
            const uint4* src = reinterpret_cast<const uint4*>(a.x + (long long)row * a.K + at);
#pragma unroll
            for (int i = 0; i < 4; ++i) u[i] = __ldcs(src + i);
        }
    };
    uint4 cur[4] = {}, nxt[4] = {};
    int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    fetch(w, cur);
    pdl_wait();
    pdl_launch_dependents();                               // after the wait: the next kernel reads the tile tables before its own
    int slots = slots_of(w);
    for (; w < n_pieces; w += warps) {
        fetch(w + warps, nxt);
        const int next_slots = slots_of(w + warps);
        float v[32];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t u[4] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[8 * i + 2 * j] = __uint_as_float(u[j] << 16);
                v[8 * i + 2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
            }
        }
        uint4 word[3];
        uint32_t scale[3];
        moe_quantize_block_x3(v, word, scale);
        const int row = w / per_row, at = (w - row * per_row) * 1024 + lane * 32;
        for (int j = 0; j < a.k; ++j) {
            const int slot = j < 32 ? __shfl_sync(kFullMask, slots, j) : __ldcg(a.pair_slot + (long long)row * a.k + j);
            if (slot < 0 || at >= a.K) continue;
            uint8_t* q = a.q + (long long)slot * (a.K >> 1) + (at >> 1);
            uint8_t* sb = a.s + (long long)slot * (a.K >> 5) + (at >> 5);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                *reinterpret_cast<uint4*>(q + t * term_q) = word[t];
                sb[t * term_s] = (uint8_t)scale[t];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) cur[i] = nxt[i];
        slots = next_slots;
    }
}

// Exponent taken out of a row whose largest magnitude is m (float bits): floor(log2 m), 0 for a row of zeros.
__device__ __forceinline__ int moe_row_exponent(uint32_t m) { return m == 0 ? 0 : min(max((int)(m >> 23) - 127, -100), 126); }

// Three E4M3 terms, of rows of this GPU.  The accumulators of the gate/up GEMM are to be within FP32 whatever the scales of x and of the
// weights, so the larger and the smaller ones are normalised: x is multiplied by 2^-(its row's exponent), and the scale bytes of a pair are
// lower by its expert's typical scale exponent, the mean of W1's and W3's, from -kAct8Down to kAct8Up (the bytes of a normalised row, 120 and
// less, leave room for that).  row_exp is the sum of the two; G gets it back before the sigmoid, U keeps it out until y is written, so that
// silu(G) * U overflows hardly before G does.  Exponents of up to kAct8Plain either way are left alone: in ordinary use row_exp is 0 and the
// gate/up epilogue has nothing to multiply (1 003 tokens of 256 experts: 490 to 494 us with no exponents at all, 508 with a multiplication for each
// value, 502 this way), and the worst of them, 16 384 products of 2^17 and 6 * 2^16, are 2^100 when squared.
// A lane takes half a block of 32, a warp 512 elements of a row in each of PIECES (one up to K 4096, two up to 8192, four), so that a row is
// read once between its maximum and its terms; a block takes as many rows as its warps cover.  The next rows and their slots are on their way
// while these are quantised.  2 K bytes of a token come in, 99 K / 32 of each of its pairs go out.  Us of the stage between two events, a warp
// for 512 elements without the maximum -> this: 2 and 64 tokens of K 4096 8.3 -> 8.5, 1 003 18.5 -> 20, 2 048 35 -> 37.6; 400 of K 6144 10 -> 12.3.
constexpr int kAct8Warps = 8, kAct8Down = 100, kAct8Up = 60, kAct8Plain = 16;
__host__ __device__ __forceinline__ int moe_act8_row_warps(int K) { return K >= 512 * kAct8Warps ? kAct8Warps : (K + 511) >> 9; }
__device__ __forceinline__ int moe_act8_plain(int e) { return abs(e) <= kAct8Plain ? 0 : e; }
template <int PIECES>
__global__ void __launch_bounds__(32 * kAct8Warps, PIECES == 1 ? 4 : PIECES == 2 ? 3 : 2) moe_act_fp8_kernel(const MoeActArgs a) {
    __shared__ uint32_t warp_max[2][kAct8Warps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row_warps = moe_act8_row_warps(a.K), rows = kAct8Warps / row_warps;      // rows of a block
    const int sub = warp / row_warps, first_warp = sub * row_warps, w = warp - first_warp;
    const int stride = (int)gridDim.x * rows;
    const long long term_q = a.n_pairs * a.K, term_s = a.n_pairs * (a.K >> 5);
    auto here = [&](int row) { return sub < rows && row < a.n_tokens; };
    auto at_of = [&](int i) { return (w + i * row_warps) * 512 + lane * 16; };
    auto fetch = [&](int row, uint4 (&u)[PIECES][2]) {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            u[i][0] = u[i][1] = make_uint4(0, 0, 0, 0);
            if (here(row) && at_of(i) < a.K) {
                const uint4* src = reinterpret_cast<const uint4*>(a.x + (long long)row * a.K + at_of(i));
                u[i][0] = __ldcs(src);
                u[i][1] = __ldcs(src + 1);
            }
        }
    };
    // slot and expert of pair j of a row; -1 for a dropped pair
    auto pair_of = [&](int row, int j) -> int2 {
        const long long p = (long long)row * a.k + j;
        return here(row) && j < a.k ? make_int2(__ldcg(a.pair_slot + p), __ldcg(a.ids + p)) : make_int2(-1, 0);
    };
    auto shift_of = [&](const int2& pair) -> int {
        if (pair.x < 0) return 0;
        const int typ = __ldcg(a.typical.typical + pair.y);
        return moe_act8_plain(min(max((((typ & 255) + (typ >> 8)) >> 1) - 127, -kAct8Down), kAct8Up));
    };
    uint4 cur[PIECES][2], nxt[PIECES][2];
    int row0 = (int)blockIdx.x * rows, buf = 0;
    fetch(row0 + sub, cur);
    pdl_wait();
    pdl_launch_dependents();                               // after the wait: the next kernel reads the tile tables before its own
    int2 pair = pair_of(row0 + sub, lane);                 // lane j: the j-th pair of the row
    int shift = shift_of(pair);
    for (; row0 < a.n_tokens; row0 += stride, buf ^= 1) {      // the same number of times in every warp of the block
        const int row = row0 + sub;
        fetch(row + stride, nxt);
        const int2 next_pair = pair_of(row + stride, lane);
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < PIECES; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t u[4] = {cur[i][h].x, cur[i][h].y, cur[i][h].z, cur[i][h].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) m = max(m, max((u[j] << 16) & 0x7fffffffu, u[j] & 0x7fff0000u));
            }
        m = __reduce_max_sync(kFullMask, m);
        if (lane == 0) warp_max[buf][warp] = m;
        __syncthreads();                                       // (two buffers: one barrier a row)
        for (int i = 0; i < row_warps && sub < rows; ++i) m = max(m, warp_max[buf][first_warp + i]);
        const int e = moe_act8_plain(moe_row_exponent(m));
        const float inv = __uint_as_float((uint32_t)(127 - e) << 23);
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            float v[16];
            uint32_t bm = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t u[4] = {cur[i][h].x, cur[i][h].y, cur[i][h].z, cur[i][h].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[8 * h + 2 * j] = __uint_as_float(u[j] << 16) * inv;
                    v[8 * h + 2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u) * inv;
                }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) bm = max(bm, __float_as_uint(v[j]) & 0x7fffffffu);
            bm = max(bm, __shfl_xor_sync(kFullMask, bm, 1));
            uint4 word[3];
            uint32_t scale[3];
            moe_quantize_e4m3x3<kE4m3BfStep>(v, bm, word, scale);
            const int at = at_of(i);
            for (int j = 0; j < a.k; ++j) {
                int slot, sh;
                if (j < 32) {
                    slot = __shfl_sync(kFullMask, pair.x, j);
                    sh = __shfl_sync(kFullMask, shift, j);
                } else {
                    const int2 p = pair_of(row, j);
                    slot = p.x;
                    sh = shift_of(p);
                }
                if (slot < 0 || at >= a.K) continue;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    *reinterpret_cast<uint4*>(a.q + t * term_q + (long long)slot * a.K + at) = word[t];
                    const int byte = scale[t] == 255 ? 255 : max((int)scale[t] - sh, 0);
                    if ((lane & 1) == 0) a.s[t * term_s + (long long)slot * (a.K >> 5) + (at >> 5)] = (uint8_t)byte;
                }
            }
        }
        if (w == 0) {
            if (pair.x >= 0) a.row_exp[pair.x] = e + shift;
            for (int j = 32 + lane; j < a.k; j += 32) {
                const int2 p = pair_of(row, j);
                if (p.x >= 0) a.row_exp[p.x] = e + shift_of(p);
            }
        }
#pragma unroll
        for (int i = 0; i < PIECES; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) cur[i][h] = nxt[i][h];
        pair = next_pair;
        shift = shift_of(pair);
    }
}

constexpr int kActRowThreads = 256;                        // threads per activation row (four rows per block)
constexpr int kActRows = kPrepThreads / kActRowThreads;
constexpr int kActMaxChunks = 16384 / 8 / kActRowThreads;  // 16-byte chunks per thread at the largest K

// Normalised fp16 (and, in the first blocks, the typical weight scale of every expert).
template <bool PEER>
__global__ void __launch_bounds__(kPrepThreads) moe_act_fp16_kernel(const MoeActArgs a, const MoePeerIn in) {
    __shared__ float red_sum[kPrepThreads / 32];
    __shared__ uint32_t red_max[kPrepThreads / 32];
    __shared__ int slots[kActRows][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int blk = blockIdx.x;
    const int scale_blocks = (a.typical.n_experts + kTypicalExperts - 1) / kTypicalExperts;
    if (blk < scale_blocks) {
        pdl_wait();
        pdl_launch_dependents();
        moe_typical_scales(a.typical, blk);
        return;
    }
    blk -= scale_blocks;

    // Rows: 256 threads each, every element read once (it stays in registers between the two passes).
    const int row_blocks = gridDim.x - scale_blocks;
    const int sub = tid / kActRowThreads, t = tid % kActRowThreads;
    const int chunks = a.K >> 3;
    bool waited = false;
    if (PEER) { pdl_wait(); pdl_launch_dependents(); waited = true; }
    for (int row0 = blk * kActRows; row0 < a.n_tokens; row0 += row_blocks * kActRows) {
        const int row = row0 + sub;
        const bool live = row < a.n_tokens && (!PEER || moe_act_wanted(a, row));
        const __nv_bfloat16* src = live ? moe_act_row<PEER>(a, in, row) : nullptr;
        uint4 v[kActMaxChunks];
#pragma unroll
        for (int i = 0; i < kActMaxChunks; ++i) {
            v[i] = make_uint4(0, 0, 0, 0);
            const int c = t + i * kActRowThreads;
            if (live && c < chunks) v[i] = __ldcs(reinterpret_cast<const uint4*>(src) + c);
        }
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < kActMaxChunks; ++i) {
            const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) m = max(m, max((u[j] << 16) & 0x7fffffffu, u[j] & 0x7fff0000u));
        }
        m = __reduce_max_sync(kFullMask, m);
        if (lane == 0) red_max[warp] = m;
        if (!waited) { pdl_wait(); pdl_launch_dependents(); waited = true; }
        if (live && t < a.k && t < 32) slots[sub][t] = __ldcg(a.pair_slot + (long long)row * a.k + t);
        asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(kActRowThreads) : "memory");
        const int w0 = sub * (kActRowThreads / 32);
#pragma unroll
        for (int w = 0; w < kActRowThreads / 32; ++w) m = max(m, red_max[w0 + w]);
        const int e = moe_row_exponent(m);
        const float inv = __uint_as_float((uint32_t)(127 - e) << 23);
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < kActMaxChunks; ++i) {
            const int c = t + i * kActRowThreads;
            if (!live || c >= chunks) continue;
            const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            __half2 h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float lo = __uint_as_float(u[j] << 16) * inv, hi = __uint_as_float(u[j] & 0xffff0000u) * inv;
                ss = fmaf(lo, lo, fmaf(hi, hi, ss));
                h[j] = __floats2half2_rn(lo, hi);
            }
            for (int j = 0; j < a.k; ++j) {
                const int slot = j < 32 ? slots[sub][j] : __ldcg(a.pair_slot + (long long)row * a.k + j);
                if (slot >= 0) reinterpret_cast<uint4*>(a.xh + (long long)slot * a.K)[c] = *reinterpret_cast<const uint4*>(h);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(kFullMask, ss, off);
        if (lane == 0) red_sum[warp] = ss;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(kActRowThreads) : "memory");
        if (t < a.k && live) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < kActRowThreads / 32; ++w) s += red_sum[w0 + w];
            const float ms = s / (float)a.K;               // mean square, at most 4
            // half the exponent, rounded down; an infinite or NaN row takes 0
            const int q = (ms > 0.f && ms <= 4.f) ? (((int)(__float_as_uint(ms) >> 23) - 127) >> 1) : 0;
            for (int j = t; j < a.k; j += kActRowThreads) {
                const int slot = __ldcg(a.pair_slot + (long long)row * a.k + j);
                if (slot >= 0) a.xexp[slot] = make_int2(e, max(q, -40));
            }
        }
    }
    if (!waited) { pdl_wait(); pdl_launch_dependents(); }
}

}  // namespace dsv4
