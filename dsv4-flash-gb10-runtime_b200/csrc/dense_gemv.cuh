// Dense M=1 GEMV over a quantized weight matrix, shared by the MXFP4 and FP8-E4M3 libraries.
//   y[n] = bf16( sum_k W[n,k] * x[k] ),  FP32 accumulation across blocks.
// The rows stream through shared memory (row_stream.cuh); per-slice partial sums meet there as well.
#pragma once

#include "row_stream.cuh"

#include <cstdio>
#include <cstdlib>
#include <utility>

namespace dsv4 {

constexpr uint32_t kDenseParts = 12 * 1024;            // partial sums of a CTA at most

struct DenseArgs {
    const __nv_bfloat16* x;
    const uint8_t* w;
    const uint8_t* s;
    int K, N;
    long long w_stride, s_stride;      // bytes per row of W / per row of the scale tensor
    __nv_bfloat16* y;
};

// MATS = 1: y = W x.
// MATS = 2: the gate / up pair of a gated FFN, act[n] = bf16( silu(clamp(g[n])) * clamp(u[n]) ), g = Wg x, u = Wu x, both
//   rounded to bf16 first (as two separate GEMV calls would leave them); rows n of both matrices travel in one stage.
//   limit_g / limit_u <= 0 switch the clamp of that operand off.
// GROUPED: blockIdx.y picks one of several independent problems stacked along the rows of W (FP8 tile scales):
//   group g multiplies rows [g N, (g+1) N) with x[g K, (g+1) K) into y[g N, (g+1) N).
// RPW rows per warp and stage, SPW slices of the reduction axis per warp.
template <class Fmt, class Sc, int MATS, int RPW, int SPW, bool GROUPED>
__global__ void __launch_bounds__(kRowThreads, 2) dense_stream_kernel(const DenseArgs a_in, const uint8_t* w2, const uint8_t* s2,
                                                                     const RowPlan p, float limit_g, float limit_u) {
    extern __shared__ __align__(128) uint8_t row_smem[];
    __shared__ RowRing ring;
    __shared__ volatile int x_asked;
    __shared__ int failed;                   // MATS = 2: a wait ran out (the clamp would turn NaN into a number)
    pdl_launch_dependents();
    DenseArgs a = a_in;
    if (GROUPED) {
        const long long grp = blockIdx.y;
        a.x += grp * a.K;
        a.w += grp * a.N * a.w_stride;
        a.s += grp * (a.N >> 7) * a.s_stride;
        a.y += grp * a.N;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r_begin = (int)((long long)a.N * blockIdx.x / gridDim.x), r_end = (int)((long long)a.N * (blockIdx.x + 1) / gridDim.x);
    const int n_local = r_end - r_begin, n_stages = (n_local + p.rows - 1) / p.rows;
    const int n_blk = a.K / Fmt::kElems;
    float* const part = reinterpret_cast<float*>(row_smem + p.off_part);                   // [MATS][n_local][n_slices]
    const uint32_t smem = smem_u32(row_smem);

    if (tid == kRowWarps * 32) row_ring_init(ring, p);
    auto produce = [&]() {
        RowPos pos;
        for (int st = 0; st < n_stages - p.withheld; ++st, pos.next(p.slots)) {
            if (!row_wait_free(ring, p, pos, 1)) break;
            const int row = st * p.rows, rows = min(p.rows, n_local - row);
            const uint32_t bar = smem_u32(&ring.full[pos.slot]), dst = smem + pos.slot * p.stage_bytes;
            const long long first = r_begin + row;
            uint32_t bytes = MATS * rows * p.row_bytes;
            if (Sc::kPerRow)
#pragma unroll
                for (int m = 0; m < MATS; ++m) bytes += row_scale_bytes(p, (m == 0 ? a.s : s2) + first * a.s_stride, n_blk, rows);
            mbar_arrive_expect_tx(bar, bytes);
#pragma unroll
            for (int m = 0; m < MATS; ++m) {
                row_copy(dst + m * p.rows * p.row_bytes, (m == 0 ? a.w : w2) + first * a.w_stride, a.w_stride, p.row_bytes, rows, bar);
                if (Sc::kPerRow)
                    row_scale_copy(p, dst + MATS * p.rows * p.row_bytes + m * p.s_area, (m == 0 ? a.s : s2) + first * a.s_stride, a.s_stride,
                                   n_blk, rows, bar);
            }
        }
    };
    // tile scales of this CTA's rows as floats: [MATS][tile rows][n_blk / 8].  Requested before the first copies: a load queues
    // behind those.
    const int tiles_k = n_blk >> 3, tile0 = r_begin >> 7, n_tr = ((r_end - 1) >> 7) - tile0 + 1, n_table = Sc::kPerRow ? 0 : MATS * n_tr * tiles_k;
    float* const table = reinterpret_cast<float*>(row_smem + p.off_table);
    auto tile_scale = [&](int i) {
        const int m = i / (n_tr * tiles_k), j = i - m * n_tr * tiles_k, tr = j / tiles_k;
        return Sc::fetch(m == 0 ? a.s : s2, (tile0 + tr) << 7, (j - tr * tiles_k) << 3, a.s_stride);
    };
    uint32_t raw = 0;
    if (tid < n_table) raw = tile_scale(tid);
    if (tid == 0) {
        x_asked = 0;
        if (MATS == 2) failed = 0;
    }
    __syncthreads();                         // barriers
    // The consumers go on without the producer: when it filled the ring before the barrier above, asking for x and the tile
    // scales waited for that (eight launches of 4096 x 4096 MXFP4 35.1 us then, 31.0 now; of 2048 x 4096 FP8 28.1, 23.8).
    if (warp == kRowWarps) {
        // weights never depend on the previous kernel in the stream: they are requested without waiting for it
        if (lane == 0) {
            if (n_local * p.row_bytes * MATS > kRowSmall) row_pause(&x_asked);
            produce();
        }
    } else {
        if (tid < n_table) table[tid] = Sc::value(raw);
        for (int i = tid + kRowWarps * 32; i < n_table; i += kRowWarps * 32) table[i] = Sc::value(tile_scale(i));
        if (!Sc::kPerRow) asm volatile("bar.sync 1, %0;" ::"n"(kRowWarps * 32) : "memory");
        pdl_wait();                          // x, and the outputs below may still be read by the kernel before
        if constexpr (Sc::kPerRow) {
            if (tid == 0) x_asked = 1;
            row_x_convert(smem + p.off_x, a.x, n_blk, tid);
            asm volatile("bar.sync 1, %0;" ::"n"(kRowWarps * 32) : "memory");
        } else if (tid == 0) {
            row_x_request(ring, smem + p.off_x, a.x, a.K * 2);
            x_asked = 1;
        }
    }
    if (warp < p.warps) {
        const int w_slices = p.warps / p.n_groups, ks0 = warp % w_slices, rg = warp / w_slices;
        int blk[SPW];
        bool ok[SPW];
#pragma unroll
        for (int q = 0; q < SPW; ++q) { blk[q] = (ks0 + q * w_slices) * 32 + lane; ok[q] = blk[q] < n_blk; }
        auto give_up = [&](int st) {
#pragma unroll 1
            for (int m = 0; m < MATS; ++m)
#pragma unroll 1
                for (int ks = ks0; ks < p.n_slices; ks += w_slices)
                    row_give_up(p, st * p.rows + rg, n_local, lane, part + m * n_local * p.n_slices + ks, p.n_slices);
            if (MATS == 2) failed = 1;
        };
        const bool got_x = Sc::kPerRow || __all_sync(kFullMask, row_wait(p, ring.x, 0, 2));
        ActBlock<Fmt> xb[SPW];
#pragma unroll
        for (int q = 0; q < SPW; ++q) {
            if constexpr (Sc::kPerRow) row_act_block(smem + p.off_x, n_blk, blk[q], ok[q], xb[q]);
            else row_act_block_bf16<Fmt>(smem + p.off_x, blk[q], ok[q], xb[q]);
            if (!ok[q]) blk[q] = 0;
            if (!got_x) xb[q].scale = row_nan();
        }
        if (MATS == 2 && !got_x) failed = 1;
        RowPos pos;
        for (int st = 0; st < n_stages; ++st) {
            if (!__all_sync(kFullMask, row_wait(p, ring.full[pos.slot], pos.round, 2))) {
                give_up(st);
                break;
            }
            const uint32_t stage = smem + pos.slot * p.stage_bytes;
            const int row = st * p.rows + rg, left = n_local - row;
            const uint32_t s_row = (uint32_t)(r_begin + st * p.rows) * (uint32_t)a.s_stride;
#pragma unroll
            for (int q = 0; q < SPW; ++q) {
                if (q > 0 && ks0 + w_slices >= p.n_slices) continue;
                // All loads first, without conditions (a branch around a row keeps the next row's loads behind its sums):
                // rows past the CTA's last hold stale bytes and their sums are dropped, lanes past the row's end read
                // block 0 against activations of zero.
                uint4 w[MATS * RPW];
                float sc[MATS * RPW];
#pragma unroll
                for (int m = 0; m < MATS; ++m)
#pragma unroll
                    for (int i = 0; i < RPW; ++i) {
                        const int r = rg + i * p.n_groups, k = m * RPW + i;
                        w[k] = lds_v4(stage + (m * p.rows + r) * p.row_bytes + blk[q] * 16);
                        if (Sc::kPerRow) {
                            const uint32_t s_addr = (uint32_t)reinterpret_cast<uintptr_t>(m == 0 ? a.s : s2) + s_row;
                            sc[k] = Sc::value(lds_u8(stage + MATS * p.rows * p.row_bytes + m * p.s_area + row_scale_offset(p, s_addr, r) + blk[q]));
                        } else {
                            sc[k] = table[(m * n_tr + ((r_begin + st * p.rows + r) >> 7) - tile0) * tiles_k + (blk[q] >> 3)];
                        }
                    }
                float v[MATS * row_pow2(RPW)] = {};
#pragma unroll
                for (int m = 0; m < MATS; ++m)
#pragma unroll
                    for (int i = 0; i < RPW; ++i) v[m * row_pow2(RPW) + i] = Fmt::dot(w[m * RPW + i], xb[q].h) * (sc[m * RPW + i] * xb[q].scale);
                row_store<RPW>(v, left, p.n_groups, lane, part + row * p.n_slices + ks0 + q * w_slices, p.n_slices, n_local * p.n_slices);
            }
            row_release(ring, p, pos, lane);
        }
    }
    __syncthreads();

    for (int t = tid; t < n_local; t += kRowThreads) {
        float g = 0.f;
        for (int s = 0; s < p.n_slices; ++s) g += part[t * p.n_slices + s];
        if (MATS == 1) {
            a.y[r_begin + t] = __float2bfloat16(g);
        } else {
            float u = 0.f;
            for (int s = 0; s < p.n_slices; ++s) u += part[(n_local + t) * p.n_slices + s];
            g = __bfloat162float(__float2bfloat16(g));
            u = __bfloat162float(__float2bfloat16(u));
            if (limit_g > 0.f) g = fminf(fmaxf(g, -limit_g), limit_g);
            if (limit_u > 0.f) u = fminf(fmaxf(u, -limit_u), limit_u);
            a.y[r_begin + t] = __float2bfloat16(failed ? row_nan() : (g / (1.0f + expf(-g))) * u);
        }
    }
}

// Several tokens and several independent groups in one launch (FP8 only: the attention projections):
//   y[t, g*N + n] = bf16( sum_k W[g*N + n, k] * x[t, g*K + k] ),   W [G*N, K], scales [G*N/128, K/128].
// G = 1 is a plain batched GEMV; G > 1 is the block-diagonal shape of the grouped output projection (one launch
// instead of G).  One token runs the grouped form of dense_stream_kernel (bit-identical to the M = 1 entry); several
// tokens run dense_mma_gemv_kernel (dense_mma_gemv.cuh), which reads every weight byte once per 8 tokens.
struct DenseMultiArgs {
    DenseArgs a;                   // group 0, token 0; a.N = rows per group
    int n_groups;
    int n_tok;
    long long x_tok, y_tok;        // elements between consecutive tokens of x / y
};

// Any alignment, any stride: one warp per row, byte loads, FP32 FMA.  Only taken when a base pointer
// or a row stride is not a multiple of 16 bytes.
template <class Fmt, class Sc>
__global__ void dense_gemv_unaligned_kernel(const DenseArgs a) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= a.N) return;
    const int n_blk = a.K / Fmt::kElems;
    const uint8_t* wrow = a.w + (long long)row * a.w_stride;
    float acc = 0.f;
    for (int blk = lane; blk < n_blk; blk += 32) {
        const float sc = Sc::value(Sc::fetch(a.s, row, blk, a.s_stride));
        const __nv_bfloat16* xp = a.x + (size_t)blk * Fmt::kElems;
        float part = 0.f;
        for (int i = 0; i < 16; ++i) {
            const uint32_t byte = wrow[(size_t)blk * 16 + i];
            if (Fmt::kElems == 32) {
                const float2 f = e2m1x2_to_float2(byte);
                part = fmaf(f.x, __bfloat162float(xp[2 * i]), part);
                part = fmaf(f.y, __bfloat162float(xp[2 * i + 1]), part);
            } else {
                part = fmaf(e4m3_to_float(byte), __bfloat162float(xp[i]), part);
            }
        }
        acc = fmaf(part, sc, acc);
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(kFullMask, acc, off);
    if (lane == 0) a.y[row] = __float2bfloat16(acc);
}

inline int dense_sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

inline bool dense_pdl_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("DSV4_B200_PDL");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1;
}

// CTAs per group: one CTA per SM over all groups (two successive launches share each SM), more where a CTA's partial sums would
// not fit.  Groups that do not divide the SMs leave a few SMs with two CTAs (rounded up; rounded down, a few SMs idle: slower still),
// and everyone waits for those: with more than kRowSmall bytes of weights per SM as many CTAs as fit two per SM are faster.  Eight
// groups of 1024 x 4096 10.2 -> 8.4 us (rounded down 11.2), twelve 13.8 -> 10.1, eight of 1024 x 1024 4.1 -> 3.6; below, one per SM is: eight
// of 512 x 512 2.5 us, with two 2.8.  Groups that divide the SMs keep one: two of 1024 x 4096 3.0 us, with two CTAs per SM 3.6.
inline long long dense_grid(const DenseArgs& a, int mats, const RowPlan& p, int n_groups) {
    const long long cap = kDenseParts / (4 * mats * p.n_slices);          // rows per CTA
    const long long sms = dense_sm_count(), need = ((long long)a.N + cap - 1) / cap;
    long long grid = (sms + n_groups - 1) / n_groups;
    if (sms % n_groups != 0 && (long long)n_groups * a.N * p.row_bytes > sms * kRowSmall && 2 * sms / n_groups > grid) grid = 2 * sms / n_groups;
    if (grid < need) grid = need;
    return grid < a.N ? grid : a.N;
}
// Needs 16-byte aligned x, weights and row strides.
template <class Fmt, class Sc, int MATS, int RPW, int SPW, bool GROUPED>
inline cudaError_t dense_stream_launch_as(const DenseArgs& a, const uint8_t* w2, const uint8_t* s2, float limit_g, float limit_u,
                                          int n_groups, cudaStream_t stream) {
    auto kernel = dense_stream_kernel<Fmt, Sc, MATS, RPW, SPW, GROUPED>;
    const int n_blk = a.K / Fmt::kElems;
    RowPlan p = row_plan(n_blk, MATS, RPW, SPW);
    const long long grid = dense_grid(a, MATS, p, n_groups);
    const int most = (int)((a.N + grid - 1) / grid);
    if (Sc::kPerRow) row_plan_scales(p, MATS, n_blk, a.s_stride, 1);
    row_plan_finish(p, Sc::kPerRow ? row_x_bytes(n_blk) : a.K * 2, 4 * MATS * most * p.n_slices, Sc::kPerRow ? 0 : 4 * MATS * (most / 128 + 3) * (n_blk / 8));
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return cudaErrorInvalidDevice;
    if (dev < 0 || dev >= 64 || !done[dev]) {
        const cudaError_t err = allow_shared(kernel, kRowSmemMost);
        if (err != cudaSuccess) return err;
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, (unsigned)n_groups);
    cfg.blockDim = dim3(kRowThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dense_pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, a, w2, s2, p, limit_g, limit_u);
}
// At most four rows per warp and stage where a stage of that stays within kRowStage, else two (as many as the rows of a CTA
// need: row_spread); FP8 rows longer than 8192 have more slices than there are warps: two per warp.
template <class Fmt, class Sc, int MATS, bool GROUPED>
inline cudaError_t dense_stream_launch(const DenseArgs& a, const uint8_t* w2, const uint8_t* s2, float limit_g, float limit_u,
                                       int n_groups, cudaStream_t stream) {
    const int n_blk = a.K / Fmt::kElems;
    if constexpr (Fmt::kElems == 16) {
        if (n_blk > 32 * kRowWarps) return dense_stream_launch_as<Fmt, Sc, MATS, 2, 2, GROUPED>(a, w2, s2, limit_g, limit_u, n_groups, stream);
    }
    const RowPlan p = row_plan(n_blk, MATS, 4, 1);
    const long long grid = dense_grid(a, MATS, p, n_groups);
    switch (row_spread((int)((a.N + grid - 1) / grid), p.n_groups, p.stage_bytes <= kRowStage ? 4 : 2)) {
        case 1: return dense_stream_launch_as<Fmt, Sc, MATS, 1, 1, GROUPED>(a, w2, s2, limit_g, limit_u, n_groups, stream);
        case 2: return dense_stream_launch_as<Fmt, Sc, MATS, 2, 1, GROUPED>(a, w2, s2, limit_g, limit_u, n_groups, stream);
        case 3: return dense_stream_launch_as<Fmt, Sc, MATS, 3, 1, GROUPED>(a, w2, s2, limit_g, limit_u, n_groups, stream);
        default: return dense_stream_launch_as<Fmt, Sc, MATS, 4, 1, GROUPED>(a, w2, s2, limit_g, limit_u, n_groups, stream);
    }
}

// Launches the aligned streaming kernel when it can, the byte-wise one otherwise.
template <class Fmt, class Sc>
inline cudaError_t dense_launch(const DenseArgs& a, cudaStream_t stream) {
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; };
    if (mis(a.x) || mis(a.w) || (a.w_stride & 15) != 0) {
        const int warps = 8;
        dense_gemv_unaligned_kernel<Fmt, Sc><<<(a.N + warps - 1) / warps, warps * 32, 0, stream>>>(a);
        return cudaGetLastError();
    }
    return dense_stream_launch<Fmt, Sc, 1, false>(a, nullptr, nullptr, 0.f, 0.f, 1, stream);
}

template <class Sc>
inline cudaError_t dense_mma_launch(const DenseMultiArgs& m, cudaStream_t stream);      // dense_mma_gemv.cuh

// Several tokens / groups: needs 16-byte aligned x, weights, row strides and token strides (cudaErrorInvalidValue
// otherwise).
template <class Sc>
inline cudaError_t dense_multi_launch(const DenseMultiArgs& m, cudaStream_t stream) {
    const DenseArgs& a = m.a;
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; };
    if (mis(a.x) || mis(a.w) || (a.w_stride & 15) != 0 || (m.x_tok & 7) != 0 || m.n_groups > 65535)
        return cudaErrorInvalidValue;
    if (m.n_tok == 1) return dense_stream_launch<Fp8Format, Sc, 1, true>(a, nullptr, nullptr, 0.f, 0.f, m.n_groups, stream);
    return dense_mma_launch<Sc>(m, stream);
}

// The gate / up pair: ag and au describe the two matrices (same K, N, x); the activation goes to ag.y.
// Needs 16-byte aligned x, weights and row strides (returns cudaErrorInvalidValue otherwise).
template <class Fmt, class Sc>
inline cudaError_t dense_dual_launch(const DenseArgs& ag, const DenseArgs& au, float limit_g, float limit_u,
                                     cudaStream_t stream) {
    auto mis = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; };
    if (mis(ag.x) || mis(ag.w) || mis(au.w) || (ag.w_stride & 15) != 0 || (au.w_stride & 15) != 0)
        return cudaErrorInvalidValue;
    return dense_stream_launch<Fmt, Sc, 2, false>(ag, au.w, au.s, limit_g, limit_u, 1, stream);
}

}  // namespace dsv4
