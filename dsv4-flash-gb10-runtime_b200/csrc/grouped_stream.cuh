// Routed-expert FFN of one token at any K_in, hidden <= 4096 (multiples of 32), as two chained kernels over the row
// streaming of row_stream.cuh; the shapes with a kernel of their own (decode_stream.cuh) do not come here.
//
//   gate/up : a CTA owns a contiguous run of (expert slot, hidden row) pairs; W1 and W3 rows of a pair travel in one stage;
//             silu(g) * u goes to the workspace as FP32.
//   down    : a CTA owns a contiguous range of output rows for ALL experts and streams them expert by expert; the
//             router-weighted sum over the experts is taken inside the CTA in a fixed order and rounded once to bf16.
// The down kernel's CTAs become resident beside the gate/up kernel's and have their first stages on the way before the
// intermediate is complete.
#pragma once

#include "grouped_args.cuh"
#include "row_stream.cuh"

namespace dsv4 {

constexpr int kGateRpw = 2, kDownRpw = 4;             // rows per warp and stage (down: at most)
constexpr uint32_t kDownParts = 12 * 1024;             // partial sums of a CTA at most

__global__ void __launch_bounds__(kRowThreads, 2) grouped_gate_stream_kernel(const GroupedArgs a, const RowPlan p) {
    extern __shared__ __align__(128) uint8_t row_smem[];
    __shared__ RowRing ring;
    __shared__ int expert[8];
    __shared__ uint32_t s_mis[2][9];                           // misalignment of an expert's W1 / W3 scales
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long total = (long long)a.E * a.H;
    const int q_begin = (int)(total * blockIdx.x / gridDim.x), q_end = (int)(total * (blockIdx.x + 1) / gridDim.x);
    const int n_local = q_end - q_begin, n_stages = (n_local + p.rows - 1) / p.rows;
    float* const part = reinterpret_cast<float*>(row_smem + p.off_part);                   // [gate, up][n_local][n_slices]
    const uint32_t smem = smem_u32(row_smem);
    const int row_s = a.K >> 5;
    // Stacked weights do not depend on the previous kernel: they are requested before waiting for it.  Picked experts do,
    // and the down kernel reads the picks early, so it may start only once this grid has waited for them.
    if (a.ids != nullptr) pdl_wait();
    pdl_launch_dependents();
    if (tid == kRowWarps * 32) row_ring_init(ring, p);
    if (tid < a.E) {
        const int id = a.ids != nullptr ? __ldcg(a.ids + tid) : tid;
        expert[tid] = id;
        s_mis[0][tid] = (uint32_t)reinterpret_cast<uintptr_t>(a.w1s + id * a.strideAs) & 15u;
        s_mis[1][tid] = (uint32_t)reinterpret_cast<uintptr_t>(a.w3s + id * a.strideAs) & 15u;
    }
    __syncthreads();

    // A stage may run over the end of one expert (p.rows <= 32 <= H): rows [0, n0) belong to expert e, the others to e + 1.
    // The scale rows of the second piece start at the next 16-byte boundary behind the first's copy.  The walk keeps (e, h) of
    // the stage's first row and takes no division: recomputing them cost half of this kernel's instructions.
    struct Walk { int e, h, n0, n1; };
    auto walk_start = [&]() { const int e = q_begin / a.H; return Walk{e, q_begin - e * a.H, 0, 0}; };
    auto walk_stage = [&](Walk& c, int st) {                   // pieces of stage st, whose first row is (e, h)
        const int rows = min(p.rows, n_local - st * p.rows);
        c.n0 = min(rows, a.H - c.h);
        c.n1 = rows - c.n0;
    };
    auto walk_next = [&](Walk& c) {
        c.h += p.rows;
        if (c.h >= a.H) { c.h -= a.H; ++c.e; }
    };
    if (warp == kRowWarps) {
        if (lane == 0) {
            RowPos pos;
            Walk c = walk_start();
            for (int st = 0; st < n_stages - p.withheld; ++st, pos.next(p.slots), walk_next(c)) {
                if (!row_wait_free(ring, p, pos, 1)) break;
                walk_stage(c, st);
                const uint32_t bar = smem_u32(&ring.full[pos.slot]), dst = smem + pos.slot * p.stage_bytes;
                uint32_t s0[2], b0[2], s1[2], b1[2], bytes = 2 * (c.n0 + c.n1) * p.row_bytes;
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    s0[m] = (s_mis[m][c.e] + c.h * row_s) & 15u;
                    b0[m] = round16(s0[m] + c.n0 * row_s);
                    s1[m] = s_mis[m][c.e + 1];
                    b1[m] = c.n1 > 0 ? round16(s1[m] + c.n1 * row_s) : 0u;
                    bytes += b0[m] + b1[m];
                }
                mbar_arrive_expect_tx(bar, bytes);
                const long long e0 = expert[c.e], e1 = c.n1 > 0 ? expert[c.e + 1] : 0;
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const uint8_t* w = m == 0 ? a.w1p : a.w3p;
                    const uint8_t* s = m == 0 ? a.w1s : a.w3s;
                    const uint32_t wd = dst + m * p.rows * p.row_bytes, sd = dst + 2 * p.rows * p.row_bytes + m * p.s_area;
                    bulk_copy_g2s(wd, w + e0 * a.strideAp + (long long)c.h * p.row_bytes, c.n0 * p.row_bytes, bar);
                    bulk_copy_g2s(sd, s + e0 * a.strideAs + (long long)c.h * row_s - s0[m], b0[m], bar);
                    if (c.n1 > 0) {
                        bulk_copy_g2s(wd + c.n0 * p.row_bytes, w + e1 * a.strideAp, c.n1 * p.row_bytes, bar);
                        bulk_copy_g2s(sd + b0[m], s + e1 * a.strideAs - s1[m], b1[m], bar);
                    }
                }
            }
        }
        __syncwarp();
        pdl_wait();
    } else {
        pdl_wait();
        row_x_convert(smem + p.off_x, a.x, row_s, tid);
        asm volatile("bar.sync 1, %0;" ::"n"(kRowWarps * 32) : "memory");
        if (warp < p.warps) {
            const int ks = warp % p.n_slices, rg = warp / p.n_slices, blk = ks * 32 + lane;
            const bool ok = blk < row_s;
            ActBlock<Fp4Format> xb;
            row_act_block(smem + p.off_x, row_s, blk, ok, xb);
            const uint32_t blk_r = ok ? blk : 0;               // lanes past the row's end: block 0 against zeros
            RowPos pos;
            Walk c = walk_start();
            for (int st = 0; st < n_stages; ++st, walk_next(c)) {
                if (!__all_sync(kFullMask, row_wait(p, ring.full[pos.slot], pos.round, 1))) {      // (NaN for the gate is enough)
                    row_give_up(p, st * p.rows + rg, n_local, lane, part + ks, p.n_slices);
                    break;
                }
                walk_stage(c, st);
                const uint32_t stage = smem + pos.slot * p.stage_bytes;
                const int row = st * p.rows + rg;
                uint4 w[2 * kGateRpw];
                float sc[2 * kGateRpw], v[2 * kGateRpw];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const uint32_t s0 = (s_mis[m][c.e] + c.h * row_s) & 15u;
                    const uint32_t second = round16(s0 + c.n0 * row_s) + s_mis[m][c.e + 1] - c.n0 * row_s;   // offset of row i of piece 1, less i row_s
                    const uint32_t sbase = stage + 2 * p.rows * p.row_bytes + m * p.s_area + blk_r;
#pragma unroll
                    for (int j = 0; j < kGateRpw; ++j) {
                        const int i = rg + j * p.n_groups;
                        w[m * kGateRpw + j] = lds_v4(stage + (m * p.rows + i) * p.row_bytes + blk_r * 16);
                        sc[m * kGateRpw + j] = e8m0_to_float_fast(lds_u8(sbase + i * row_s + (i < c.n0 || c.n1 == 0 ? s0 : second)));
                    }
                }
#pragma unroll
                for (int k = 0; k < 2 * kGateRpw; ++k) v[k] = Fp4Format::dot(w[k], xb.h) * (sc[k] * xb.scale);
                row_store<kGateRpw>(v, n_local - row, p.n_groups, lane, part + row * p.n_slices + ks, p.n_slices, n_local * p.n_slices);
                row_release(ring, p, pos, lane);
            }
        }
    }
    __syncthreads();
    for (int t = tid; t < n_local; t += kRowThreads) {
        float g = 0.f, u = 0.f;
        for (int s = 0; s < p.n_slices; ++s) { g += part[t * p.n_slices + s]; u += part[(n_local + t) * p.n_slices + s]; }
        a.mid[q_begin + t] = swiglu_f32(g, u);
    }
}

// early_ids: the launch before this one is the gate/up kernel of the same call, so the picks may be read before waiting.
// RPW: rows per warp and stage (row_spread).
template <int RPW>
__global__ void __launch_bounds__(kRowThreads, 2) grouped_down_stream_kernel(const GroupedArgs a, const RowPlan p, int early_ids) {
    extern __shared__ __align__(128) uint8_t row_smem[];
    __shared__ RowRing ring;
    __shared__ int expert[8];
    __shared__ float weight[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int o_begin = (int)((long long)a.O * blockIdx.x / gridDim.x), o_end = (int)((long long)a.O * (blockIdx.x + 1) / gridDim.x);
    const int n_local = o_end - o_begin, per_e = (n_local + p.rows - 1) / p.rows, n_stages = a.E * per_e;
    const int n_blk = a.H >> 5;
    uint4* const mid = reinterpret_cast<uint4*>(row_smem + p.off_x);                                   // [E][n_blk][4], chunks rotated
    float* const mid_scale = reinterpret_cast<float*>(mid + (size_t)a.E * n_blk * 4);                  // [E][n_blk]
    float* const part = reinterpret_cast<float*>(row_smem + p.off_part);                               // [n_local][E][n_slices]
    const uint32_t smem = smem_u32(row_smem);
    pdl_launch_dependents();
    if (a.ids != nullptr && !early_ids) pdl_wait();
    if (tid == kRowWarps * 32) row_ring_init(ring, p);
    if (tid < a.E) expert[tid] = a.ids != nullptr ? __ldcg(a.ids + tid) : tid;
    __syncthreads();
    auto scales_of = [&](int e, int row) { return a.w2s + (long long)expert[e] * a.strideBs + (long long)(o_begin + row) * n_blk; };
    if (warp == kRowWarps) {
        if (lane == 0) {
            RowPos pos;
            for (int st = 0; st < n_stages - p.withheld; ++st, pos.next(p.slots)) {
                if (!row_wait_free(ring, p, pos, 2)) break;
                const int e = st / per_e, row = (st - e * per_e) * p.rows, rows = min(p.rows, n_local - row);
                const uint32_t bar = smem_u32(&ring.full[pos.slot]), dst = smem + pos.slot * p.stage_bytes;
                const uint8_t* s = scales_of(e, row);
                mbar_arrive_expect_tx(bar, rows * p.row_bytes + row_scale_bytes(p, s, n_blk, rows));
                bulk_copy_g2s(dst, a.w2p + (long long)expert[e] * a.strideBp + (long long)(o_begin + row) * p.row_bytes, rows * p.row_bytes, bar);
                row_scale_copy(p, dst + p.rows * p.row_bytes, s, n_blk, n_blk, rows, bar);
            }
        }
        __syncwarp();
        pdl_wait();
    } else {
        pdl_wait();
        if (tid < a.E) weight[tid] = __ldcg(a.r + tid);
        // The intermediate of every expert -> fp16 blocks with a power of two each; chunk c of block b at (c + (b >> 1)) & 3,
        // so that lanes reading the same chunk of neighbouring blocks meet in no bank.  Eight lanes share a block (four
        // values each) and a thread has four pieces in flight: with a block per thread the loads were 128 bytes apart, and
        // every CTA of the grid asking for the same lines that way cost this kernel 4 us of L2 time.
        constexpr int kPieces = 4;
        const int n_pieces = a.E * n_blk * 8;
        for (int base = 0; base < n_pieces; base += kRowWarps * 32 * kPieces) {      // the same trips for every thread: lanes exchange
            const int i0 = base + tid;
            float4 f[kPieces];
#pragma unroll
            for (int u = 0; u < kPieces; ++u) {
                const int i = i0 + u * kRowWarps * 32;
                f[u] = i < n_pieces ? __ldcg(reinterpret_cast<const float4*>(a.mid) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < kPieces; ++u) {
                const int i = i0 + u * kRowWarps * 32, b = i >> 3, q = i & 7;
                uint32_t m = max(max(__float_as_uint(f[u].x) & 0x7fffffffu, __float_as_uint(f[u].y) & 0x7fffffffu),
                                 max(__float_as_uint(f[u].z) & 0x7fffffffu, __float_as_uint(f[u].w) & 0x7fffffffu));
#pragma unroll
                for (int off = 1; off < 8; off <<= 1) m = max(m, __shfl_xor_sync(kFullMask, m, off));
                const int e = min(max((int)(m >> 23) - Fp4Format::kActExp, 1), 253);
                const float inv = __uint_as_float((uint32_t)(254 - e) << 23);
                const __half2 lo = __floats2half2_rn(f[u].x * inv, f[u].y * inv), hi = __floats2half2_rn(f[u].z * inv, f[u].w * inv);
                if (i < n_pieces) {
                    reinterpret_cast<uint2*>(mid)[(b * 4 + (((q >> 1) + (b >> 1)) & 3)) * 2 + (q & 1)] =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                    if (q == 0) mid_scale[b] = __uint_as_float((uint32_t)e << 23);
                }
            }
        }
        // the consumers only: the producer is waiting for them to empty its ring
        asm volatile("bar.sync 1, %0;" ::"n"(kRowWarps * 32) : "memory");
        if (warp < p.warps) {
            const int ks = warp % p.n_slices, rg = warp / p.n_slices, blk = ks * 32 + lane;
            const bool ok = blk < n_blk;
            ActBlock<Fp4Format> xb;
            RowPos pos;
            bool alive = true;
            const int blk_r = ok ? blk : 0;
            for (int e = 0; e < a.E && alive; ++e) {
                {
                    const int b = e * n_blk + blk_r;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint4 q = mid[b * 4 + ((c + (b >> 1)) & 3)];
                        if (!ok) q = make_uint4(0, 0, 0, 0);
                        *reinterpret_cast<uint4*>(&xb.h[4 * c]) = q;
                    }
                    xb.scale = mid_scale[b];
                }
                const uint32_t s_first = (uint32_t)reinterpret_cast<uintptr_t>(scales_of(e, 0));
                for (int row0 = 0; row0 < n_local; row0 += p.rows) {
                    if (!__all_sync(kFullMask, row_wait(p, ring.full[pos.slot], pos.round, 2))) {      // (the last expert's product is enough)
                        row_give_up(p, (e == a.E - 1 ? row0 : 0) + rg, n_local, lane, part + (a.E - 1) * p.n_slices + ks, a.E * p.n_slices);
                        alive = false;
                        break;
                    }
                    const uint32_t stage = smem + pos.slot * p.stage_bytes, sbase = stage + p.rows * p.row_bytes + blk_r;
                    const uint32_t s_addr = s_first + row0 * n_blk;
                    const int row = row0 + rg;
                    uint4 w[RPW];
                    float sc[RPW], v[row_pow2(RPW)] = {};
#pragma unroll
                    for (int j = 0; j < RPW; ++j) {
                        const int i = rg + j * p.n_groups;
                        w[j] = lds_v4(stage + i * p.row_bytes + blk_r * 16);
                        sc[j] = e8m0_to_float_fast(lds_u8(sbase + row_scale_offset(p, s_addr, i)));
                    }
#pragma unroll
                    for (int j = 0; j < RPW; ++j) v[j] = Fp4Format::dot(w[j], xb.h) * (sc[j] * xb.scale);
                    row_store<RPW>(v, n_local - row, p.n_groups, lane, part + (row * a.E + e) * p.n_slices + ks, a.E * p.n_slices, 0);
                    row_release(ring, p, pos, lane);
                }
            }
        }
    }
    __syncthreads();
    for (int t = tid; t < n_local; t += kRowThreads) {
        float acc = 0.f;
        for (int k = 0; k < a.E; ++k) {
            float v = 0.f;
            for (int s = 0; s < p.n_slices; ++s) v += part[(t * a.E + k) * p.n_slices + s];
            acc = fmaf(weight[k], v, acc);
        }
        a.out[o_begin + t] = __float2bfloat16(acc);
    }
}

}  // namespace dsv4
