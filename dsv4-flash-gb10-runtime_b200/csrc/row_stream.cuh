// Row streaming through shared memory, shared by the dense GEMVs and the routed-expert FFN of one token.
//
// A CTA owns a contiguous range of weight rows.  One producer thread brings them in with bulk copies (cp.async.bulk, a
// stage of whole rows and their scale bytes), up to kRowSlots stages ahead; sixteen consumer warps take a stage together: a
// warp owns one slice of 32 16-byte blocks of the reduction axis (a lane one block of it) and every n_groups-th row, so its
// activations stay in 8 or 16 registers.
//
// What bounds it: HBM, and the chain of one launch after another.  The products need x, so they all come after the wait
// for the previous kernel; what can come before is the loading.  Loads into registers (the form before this one: 256
// threads x 126 registers) filled the register file, so the next launch of a chain could not become resident and every
// launch paid the whole ramp.  A CTA takes less than half of the SM's registers and shared memory here: under programmatic
// dependent launch the next kernel's CTAs sit beside these and have their first ~90 KB per SM (13 MB) on the way while
// these finish.  Nothing is loaded by the consumers inside the loop: a load queues behind the SM's own weight copies, one to
// four microseconds (scale bytes fetched that way, two stages ahead, made 33.6 MB of FP8 take 11.1 us).
//
// Every wait has a poll budget.  A consumer warp whose wait runs out records a status, writes NaN for its share of the rows it did
// not get and stops, without freeing another slot.  Nothing is requested past the ring then, and what was requested landed long
// before the last role has given up: no copy is on its way when the CTA leaves.  (A flag for the whole CTA, looked at behind the
// last stage, made every launch 0.05 to 0.1 us longer.)
#pragma once

#include "gemv_engine.cuh"
#include "stream_ring.cuh"

namespace dsv4 {

constexpr int kRowWarps = 16;                          // consumer warps
constexpr int kRowThreads = (kRowWarps + 1) * 32;
constexpr int kRowSlots = 8;                           // stages at most
constexpr uint32_t kRowStage = 32 * 1024;              // weight bytes of one stage, where four rows per warp fit that
constexpr uint32_t kRowSmem = 111 * 1024;              // dynamic shared memory of a CTA: two fit an SM
constexpr uint32_t kRowSmemMost = 220 * 1024;          // taken where two stages would not fit otherwise

__host__ __device__ __forceinline__ uint32_t round16(uint32_t v) { return (v + 15u) & ~15u; }

// How a matrix of n_blk 16-byte blocks per row is cut up.  Slices beyond the 16 warps (FP8 rows longer than 8192) are taken
// two per warp.
struct RowPlan {
    int n_slices, n_groups, warps;                     // warps that take part
    int rows;                                          // rows per stage (of each matrix)
    int slots;
    uint32_t row_bytes, stage_bytes;
    // scale bytes of the rows (MXFP4), behind the stage's weights: s_area bytes per matrix, see row_scale_offset
    uint32_t s_area, s_pitch, s_adv;
    uint32_t off_x, off_part, off_table;               // behind the ring
    uint32_t smem;
    uint32_t polls;                                    // budget of a wait
    int withheld;                                      // stages at a CTA's end that its producer does not request (0; see row_wait_limits)
};
// What the next launches of this library take: the poll budget of their waits, and the stages a test withholds so that waits run
// out without a fault.
static uint32_t g_row_polls = kSpinLimit;
static int g_row_withheld = 0;
inline int row_wait_limits(long long polls, int withheld) {
    if (polls < 0 || withheld < 0) return -1;
    g_row_polls = polls == 0 || polls > (long long)kSpinLimit ? kSpinLimit : (uint32_t)polls;
    g_row_withheld = withheld;
    return 0;
}
// The bytes of a stage's scale rows are copied with the 16-byte chunks they lie in (such a chunk never leaves the memory page
// of its bytes).  Rows dense in memory: one copy, row i at i * s_pitch behind the first; otherwise a copy per row, each with
// its own misalignment.
__device__ __forceinline__ uint32_t row_scale_offset(const RowPlan& p, uint32_t addr0, int i) {
    return (uint32_t)i * p.s_pitch + ((addr0 + (uint32_t)i * p.s_adv) & 15u);
}
// rpw: rows per warp and stage, spw: slices per warp, mats: matrices streamed side by side
inline RowPlan row_plan(int n_blk, int mats, int rpw, int spw) {
    RowPlan p = {};
    p.polls = g_row_polls;
    p.withheld = g_row_withheld;
    p.n_slices = (n_blk + 31) / 32;
    const int w = (p.n_slices + spw - 1) / spw;
    p.n_groups = kRowWarps / w;
    p.warps = w * p.n_groups;
    p.row_bytes = (uint32_t)n_blk * 16u;
    p.rows = rpw * p.n_groups;
    p.stage_bytes = (uint32_t)mats * p.rows * p.row_bytes;
    return p;
}
// row_s scale bytes per row, stride bytes from row to row; `pieces` runs of rows that are apart in memory
inline void row_plan_scales(RowPlan& p, int mats, uint32_t row_s, long long stride, int pieces) {
    const bool dense = stride == (long long)row_s;
    p.s_pitch = dense ? row_s : round16(row_s) + 16;
    p.s_adv = dense ? 0u : (uint32_t)(stride & 15);
    p.s_area = (dense ? round16(p.rows * row_s) : p.rows * p.s_pitch) + 32u * pieces;
    p.stage_bytes += mats * p.s_area;
}
// Ring depth and offsets: x_bytes of activations, part_bytes of partial sums, table_bytes of tile scales behind the ring.
inline void row_plan_finish(RowPlan& p, uint32_t x_bytes, uint32_t part_bytes, uint32_t table_bytes) {
    const uint32_t rest = round16(x_bytes) + round16(part_bytes) + round16(table_bytes);
    uint32_t most = kRowSmem;
    if (rest + 2 * p.stage_bytes > most) most = kRowSmemMost;
    const int fit = (int)((most - rest) / p.stage_bytes);
    p.slots = fit < kRowSlots ? fit : kRowSlots;
    p.off_x = p.slots * p.stage_bytes;
    p.off_part = p.off_x + round16(x_bytes);
    p.off_table = p.off_part + round16(part_bytes);
    p.smem = p.off_table + round16(table_bytes);
}

// Scales.  Per row and block (MXFP4): they travel with the rows.  Per 128 x 128 tile (FP8): a table in shared memory.
struct Fp4Scale {   // E8M0 [N, K/32]: one byte per row per block
    static constexpr bool kPerRow = true;
    __device__ static __forceinline__ uint32_t fetch(const uint8_t* s, int row, int blk, long long s_stride) {
        return ldg_stream_u8(s + (long long)row * s_stride + blk);
    }
    __device__ static __forceinline__ float value(uint32_t raw) { return e8m0_to_float(raw); }
};
struct Fp8Scale {   // E8M0 [N/128, K/128]: one byte per 128x128 tile; a block is 16 elements
    static constexpr bool kPerRow = false;
    __device__ static __forceinline__ uint32_t fetch(const uint8_t* s, int row, int blk, long long s_stride) {
        return ldg_stream_u8(s + (long long)(row >> 7) * s_stride + (blk >> 3));
    }
    __device__ static __forceinline__ float value(uint32_t raw) { return e8m0_to_float(raw); }
};
struct Fp8ScaleF32 {   // FP32 [N/128, K/128], row stride in bytes
    static constexpr bool kPerRow = false;
    __device__ static __forceinline__ uint32_t fetch(const uint8_t* s, int row, int blk, long long s_stride) {
        return __ldg(reinterpret_cast<const uint32_t*>(s + (long long)(row >> 7) * s_stride) + (blk >> 3));
    }
    __device__ static __forceinline__ float value(uint32_t raw) { return __uint_as_float(raw); }
};

// Rows per warp and stage where at most `most` fit: a CTA's `rows` spread evenly over its stages.  The warps' instructions bound
// short launches (a stage of four rows per warp is 1.1 us of them, whatever rows there are): six experts of 2880 x 1440 19.1 ->
// 17.5 us, of 1024 x 544 13.2 -> 9.4.
inline int row_spread(int rows, int n_groups, int most) {
    const int stages = (rows + most * n_groups - 1) / (most * n_groups);
    return (rows + stages * n_groups - 1) / (stages * n_groups);
}

// Dynamic shared memory of a kernel, and the SM's memory split for the most shared memory.  The split follows a kernel's own
// needs otherwise, and an SM changes it only when it is empty: launches with different needs then do not overlap
// (eight shared experts of 1536, 1152: 48.4 -> 38.5 us).
template <class Kernel>
inline cudaError_t allow_shared(Kernel kernel, size_t bytes) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err != cudaSuccess) return err;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

// The barriers of a CTA: the ring's, and one for x.
struct RowRing {
    uint64_t full[kRowSlots], empty[kRowSlots], x;
};
__device__ __forceinline__ void row_ring_init(RowRing& r, const RowPlan& p) {
    for (int s = 0; s < p.slots; ++s) { mbar_init(smem_u32(&r.full[s]), 1); mbar_init(smem_u32(&r.empty[s]), p.warps); }
    mbar_init(smem_u32(&r.x), 1);
    mbar_init_fence();
}
struct RowPos {
    int slot = 0;
    uint32_t round = 0;
    __device__ __forceinline__ void next(int n) { if (++slot == n) { slot = 0; ++round; } }
};
// Waits for a phase; the budget is looked at only where a wait is a long one.
__device__ __forceinline__ bool row_wait(const RowPlan& p, uint64_t& bar, uint32_t parity, int code) {
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(smem_u32(&bar), parity & 1u)) return true;
        if (it > 64) {
            __nanosleep(64);
            if (it >= p.polls) break;
        }
    }
    atomicExch(&g_device_status, code);
    return false;
}
// The producer's wait for a free slot.  The consumers free nothing before the previous kernel's end, which may be any time away:
// that wait comes first and is not part of the budget.
__device__ __forceinline__ bool row_wait_free(RowRing& r, const RowPlan& p, const RowPos& pos, int code) {
    if (pos.round == 0) return true;
    if (pos.round == 1 && pos.slot == 0) pdl_wait();
    return row_wait(p, r.empty[pos.slot], pos.round - 1, code);
}
__device__ __forceinline__ float row_nan() { return __uint_as_float(0x7fffffffu); }
// NaN for a warp's rows from `first` on (its every n_groups-th), by its lanes.
__device__ __forceinline__ void row_give_up(const RowPlan& p, int first, int n_local, int lane, float* part, int part_stride) {
    for (int t = first + lane * p.n_groups; t < n_local; t += 32 * p.n_groups) part[t * part_stride] = row_nan();
}
__device__ __forceinline__ void row_release(RowRing& r, const RowPlan& p, RowPos& pos, int lane) {
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&r.empty[pos.slot])) : "memory");
    pos.next(p.slots);
}

// `rows` weight rows from `src` to shared memory, dense there: one copy where they are dense in memory.  Returns the bytes.
__device__ __forceinline__ void row_copy(uint32_t dst, const uint8_t* src, long long stride, uint32_t row_bytes, int rows, uint32_t bar) {
    if (stride == (long long)row_bytes) {
        bulk_copy_g2s(dst, src, rows * row_bytes, bar);
    } else {
        for (int i = 0; i < rows; ++i) bulk_copy_g2s(dst + i * row_bytes, src + i * stride, row_bytes, bar);
    }
}
// Bytes that the copies of `rows` scale rows at `src` bring in, and the copies.
__device__ __forceinline__ uint32_t row_scale_bytes(const RowPlan& p, const uint8_t* src, uint32_t row_s, int rows) {
    const uint32_t a = (uint32_t)reinterpret_cast<uintptr_t>(src);
    if (p.s_pitch == row_s) return round16((a & 15u) + rows * row_s);
    uint32_t sum = 0;
    for (int i = 0; i < rows; ++i) sum += round16(((a + i * p.s_adv) & 15u) + row_s);
    return sum;
}
__device__ __forceinline__ void row_scale_copy(const RowPlan& p, uint32_t dst, const uint8_t* src, long long stride, uint32_t row_s, int rows,
                                               uint32_t bar) {
    if (p.s_pitch == row_s) {
        const uint32_t mis = (uint32_t)reinterpret_cast<uintptr_t>(src) & 15u;
        bulk_copy_g2s(dst, src - mis, round16(mis + rows * row_s), bar);
    } else {
        for (int i = 0; i < rows; ++i) {
            const uint8_t* at = src + i * stride;
            const uint32_t mis = (uint32_t)reinterpret_cast<uintptr_t>(at) & 15u;
            bulk_copy_g2s(dst + i * p.s_pitch, at - mis, round16(mis + row_s), bar);
        }
    }
}

// Activations, FP8: a bulk copy of x, and a lane converts its block.
template <class Fmt>
__device__ __forceinline__ void row_act_block_bf16(uint32_t x_smem, int blk, bool valid, ActBlock<Fmt>& a) {
    float v[Fmt::kElems];
#pragma unroll
    for (int i = 0; i < Fmt::kElems / 8; ++i) {
        uint4 q = make_uint4(0, 0, 0, 0);
        if (valid) q = lds_v4(x_smem + (uint32_t)blk * (Fmt::kElems * 2) + 16 * i);
        const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[8 * i + 2 * j + 0] = __uint_as_float(u[j] << 16);
            v[8 * i + 2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
        }
    }
    act_block_finish<Fmt>(v, a);
}
// x (bf16, 16-byte aligned, a multiple of 16 bytes) -> shared memory, once per CTA, by one thread after its pdl_wait: every
// warp reading its slice from global memory put 600 readers on each line of x, half a microsecond of L2 time.
__device__ __forceinline__ void row_x_request(RowRing& r, uint32_t x_smem, const __nv_bfloat16* x, uint32_t bytes) {
    mbar_arrive_expect_tx(smem_u32(&r.x), bytes);
    bulk_copy_g2s(x_smem, x, bytes, smem_u32(&r.x));
}
// Activations, MXFP4: x (bf16, 16-byte aligned) -> shared memory as fp16 blocks with a power of two each, once per CTA, by the
// consumers after their pdl_wait; four lanes share a block.  A block is 32 values here, and every warp converting its own cost half
// a microsecond of a launch: eight launches of 10007 x 2912 46.7 -> 43.0 us, of 1000 x 1024 19.1 -> 16.7.  (FP8 blocks are 16
// values: eight launches of 2048 x 4096 took 23.8 us with the copy and 24.6 this way.)  A barrier of the consumers must follow.  Chunks of a block are placed so that lanes reading the same chunk of neighbouring blocks meet in no bank.
__device__ __forceinline__ uint32_t row_x_chunk(int blk, int c) { return (uint32_t)blk * 4 + ((c + (blk >> 1)) & 3); }
__host__ __device__ __forceinline__ uint32_t row_x_bytes(int n_blk) { return (uint32_t)n_blk * 68; }
__device__ __forceinline__ void row_x_convert(uint32_t x_smem, const __nv_bfloat16* x, int n_blk, int tid) {
    constexpr int kPieces = 2;
    const int n = n_blk * 4;
    for (int base = 0; base < n; base += kPieces * kRowWarps * 32) {          // the same trips for every thread: lanes exchange
        uint4 q[kPieces];
#pragma unroll
        for (int u = 0; u < kPieces; ++u) {
            const int i = base + u * kRowWarps * 32 + tid;
            q[u] = i < n ? __ldcg(reinterpret_cast<const uint4*>(x) + i) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < kPieces; ++u) {
            const int i = base + u * kRowWarps * 32 + tid, b = i >> 2, c = i & 3;
            if (base + u * kRowWarps * 32 >= n) break;
            const uint32_t w[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
            uint32_t m = 0, h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) m = max(m, max(w[j] & 0x7fffu, (w[j] >> 16) & 0x7fffu));
#pragma unroll
            for (int off = 1; off < 4; off <<= 1) m = max(m, __shfl_xor_sync(kFullMask, m, off));
            const int e = min(max((int)(m >> 7) - Fp4Format::kActExp, 1), 253);     // biased exponent of the scale
            const float inv = __uint_as_float((uint32_t)(254 - e) << 23);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 p = __floats2half2_rn(__uint_as_float(w[j] << 16) * inv, __uint_as_float(w[j] & 0xffff0000u) * inv);
                h[j] = *reinterpret_cast<const uint32_t*>(&p);
            }
            if (i < n) {
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(x_smem + row_x_chunk(b, c) * 16),
                             "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
                if (c == 0) asm volatile("st.shared.b32 [%0], %1;" ::"r"(x_smem + (uint32_t)n * 16 + b * 4), "r"((uint32_t)e << 23) : "memory");
            }
        }
    }
}
__device__ __forceinline__ void row_act_block(uint32_t x_smem, int n_blk, int blk, bool valid, ActBlock<Fp4Format>& a) {
    const int b = valid ? blk : 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint4 q = lds_v4(x_smem + row_x_chunk(b, c) * 16);
        if (!valid) q = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(&a.h[4 * c]) = q;
    }
    uint32_t s;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(s) : "r"(x_smem + (uint32_t)n_blk * 64 + b * 4));
    a.scale = __uint_as_float(s);
}

// Before the first copies of a CTA: the previous launch's CTA on this SM asks for its activations about when this one starts (a
// third CTA has just made room for it), and behind a full ring they come a microsecond late.  So a ring of more than kRowSmall
// bytes waits kRowPause clocks, unless this CTA's own activations have been asked for (nothing runs before it).  Eight launches of
// 10007 x 2912 MXFP4 50.2 -> 48.5 us, eight of 8192 x 4096 FP8 65.5 -> 63.7 us; smaller rings lose by waiting (6000 x 1600: 30.8 -> 32.8).
constexpr uint32_t kRowSmall = 40 * 1024;
constexpr int kRowPause = 800;
__device__ __forceinline__ void row_pause(const volatile int* x_asked) {
    const long long t0 = clock64();
    while (clock64() - t0 < kRowPause && !*x_asked) { }
}

// Sums over the lanes of a warp's rows of one stage: v[m * row_pow2(RPW) + i], i < RPW, is row i * n_groups of matrix m, and goes
// to part[m * mat_stride + i * n_groups * part_stride] (one writer per row).
__host__ __device__ constexpr int row_pow2(int rpw) { return rpw == 3 ? 4 : rpw; }
template <int RPW, int V>
__device__ __forceinline__ void row_store(float (&v)[V], int rows_left, int n_groups, int lane, float* part, int part_stride, int mat_stride) {
    multi_reduce<V>(v, lane);
    if (multi_reduce_owner<V>(lane)) {
        constexpr int P = row_pow2(RPW);
        const int k = multi_reduce_index<V>(lane), i = k % P;
        if (i < RPW && i * n_groups < rows_left) part[(V > P ? k / P * mat_stride : 0) + i * n_groups * part_stride] = v[0];
    }
}

}  // namespace dsv4
