// libmxfp4_moe.so — routed-expert MXFP4 MoE layer for a BATCH of tokens on B200 (sm_100a): batched decode and
// prefill.  No counterpart in the reference (its path is one token at a time,
// runtime/dsv4_engine_mxfp4.py:412-422 loops tokens); the arithmetic contract is the same FFN:
//   out[t] = sum_j w[t, j] * W2_e ( silu(W1_e x_t) * (W3_e x_t) ),  e = ids[t, j].
// Pipeline on the caller's stream: pairs grouped by expert; grouped GEMM 1 (gate/up + SwiGLU) and grouped GEMM 2
// (down, router weight applied) on tcgen05 tensor cores; per-token sum in the router's order.  Two tensor-core
// paths: block-scaled MXFP4 MMAs fed with the packed weights as stored (moe_gemm_mxf4.cuh; activations as three
// MXFP4 terms; the default), and "fp16" for more precise activations: the same kernel with three E4M3 terms, or fp16 MMAs with the
// weights dequantised into tensor memory (moe_gemm_kernel.cuh).
// Nothing is allocated; all scratch lives in the caller's workspace.
#include "moe_gemm_kernel.cuh"
#include "moe_prep_kernel.cuh"
#include "moe_gemm_mxf4.cuh"
#include "moe_mma_rate.cuh"

#include <cstdio>
#include <cstdlib>

using namespace dsv4;

namespace {

struct Carve {
    size_t off = 0;
    size_t take(size_t bytes) { const size_t at = off; off += (bytes + 255) & ~size_t(255); return at; }
};

struct WorkspaceMap {
    size_t offsets, tiles_up, tiles_down, pair_slot, slot_w, y;      // both paths
    size_t xq, xs, mq, ms;                                          // block-scaled path
    size_t xh, xexp, typical, mid, mid_exp;                         // fp16 path (the same bytes)
    size_t xq8, xs8, mq8, ms8, row_exp8, typical8;                  // its form on the block-scaled MMAs (the same bytes; x in those of y)
    bool fits8;                                                     // which hold it
    size_t total;
};

WorkspaceMap map_workspace(long long T, int k, int K, int H, int O, int E) {
    const long long P = T * k;
    Carve c;
    WorkspaceMap m;
    m.offsets = c.take((size_t)(E + 1) * 4);
    m.tiles_up = c.take((size_t)(E + 1) * 4);
    m.tiles_down = c.take((size_t)(E + 1) * 4);
    m.pair_slot = c.take((size_t)P * 4);
    m.slot_w = c.take((size_t)P * 4);
    m.y = c.take((size_t)P * O * 4);
    const size_t shared = c.off;
    // three MXFP4 terms of x (a row per pair) and of the intermediate
    m.xq = c.take((size_t)3 * P * K / 2);
    m.xs = c.take((size_t)3 * P * K / 32);
    m.mq = c.take((size_t)3 * P * H / 2);
    m.ms = c.take((size_t)3 * P * H / 32);
    const size_t mxf4_end = c.off;
    c.off = shared;
    m.xh = c.take((size_t)P * K * 2);
    m.xexp = c.take((size_t)P * 8);
    m.typical = c.take((size_t)E * 4);
    m.mid = c.take((size_t)P * H * 2);
    m.mid_exp = c.take((size_t)P * 4);
    m.total = c.off > mxf4_end ? c.off : mxf4_end;
    // three E4M3 terms: x is done with before the down GEMM writes y
    c.off = m.y;
    m.xq8 = c.take((size_t)3 * P * K);
    m.xs8 = c.take((size_t)3 * P * K / 32);
    m.fits8 = c.off <= shared;
    c.off = shared;
    m.mq8 = c.take((size_t)3 * P * H);
    m.ms8 = c.take((size_t)3 * P * H / 32);
    m.row_exp8 = c.take((size_t)P * 4);
    m.typical8 = c.take((size_t)E * 4);
    m.fits8 = m.fits8 && c.off <= m.total;
    return m;
}

int sm_count() {
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

// Per function and device, once: `bytes` is the most that any shape needs.  (With the bytes of the call, two threads with
// different numbers of experts could leave the smaller of the two set.)
template <class Kernel>
cudaError_t allow_smem(Kernel kernel, size_t bytes, int (&done)[64]) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (done[dev] >= (int)bytes) return cudaSuccess;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err == cudaSuccess) done[dev] = (int)bytes;
    return err;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// DSV4_B200_PDL=0 switches programmatic dependent launch off (debugging).
bool pdl_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("DSV4_B200_PDL");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1;
}

// Consecutive kernels are launched with programmatic stream serialisation: a kernel's CTAs are scheduled while the one before it
// drains, and what they do before griddepcontrol.wait (barrier set-up, tensor memory allocation, first reads) overlaps its tail.
// What a kernel may read before its wait follows from when the one before it triggers (griddepcontrol.launch_dependents):
//   * A kernel that triggers only AFTER its own wait tells its successor that everything before itself is complete.  That holds
//     for the grouping kernel (behind it the activation kernels read x), the activation kernels (behind them the gate/up GEMM reads
//     the tile tables and requests weights) and the gate/up GEMM (behind it the down GEMM does).  Their triggers must stay there.
//   * The combine kernels, moe_ep_gather_meta_kernel and moe_ep_sum_kernel trigger first; what follows them (the grouping
//     kernel, or another call) reads nothing of theirs, nor of what is before them, until its own wait.
// Every kernel writes global memory only after its wait.
template <class... Params, class... Args>
cudaError_t launch_k(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                     Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Row-major tensors seen in boxes of 128 bytes of the innermost axis, 128-byte swizzle.  The encoder is a
// driver function without side effects on the device; it is looked up once.
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
cudaError_t box_map(CUtensorMap* map, CUtensorMapDataType type, int row_bytes, const void* base, int rank, const cuuint64_t* dim,
                    const cuuint32_t* box) {
    static EncodeTiled encode = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &res) != cudaSuccess) p = nullptr;
        return reinterpret_cast<EncodeTiled>(p);
    }();
    if (!encode) return cudaErrorNotSupported;
    const cuuint64_t stride[2] = {(cuuint64_t)row_bytes, (cuuint64_t)row_bytes * dim[1]};
    const cuuint32_t step[3] = {1, 1, 1};
    const CUresult r = encode(map, type, (cuuint32_t)rank, const_cast<void*>(base), dim, stride, box, step,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
// packed weights [rows, K / 2]: 128 rows
cudaError_t weight_map(CUtensorMap* map, const uint8_t* base, long long rows, int K) {
    const cuuint64_t dim[2] = {(cuuint64_t)(K / 2), (cuuint64_t)rows};
    const cuuint32_t box[2] = {128, kMoeTileRows};
    return box_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, K / 2, base, 2, dim, box);
}
// the same laid down in groups of 8 bytes and 8 of padding: 128 elements a row (base 32-byte aligned)
cudaError_t weight_map_padded(CUtensorMap* map, const uint8_t* base, long long rows, int K) {
    const cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint32_t box[2] = {128, kMoeTileRows};
    return box_map(map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, K / 2, base, 2, dim, box);
}
// three terms [3][P][row_bytes]: half a tile's columns of every term; boxes of the column counts that tiles of up to `cap` tokens have
cudaError_t term_maps(CUtensorMap (&map)[kMoeWidths], const uint8_t* base, long long P, int row_bytes, int cap) {
    cudaError_t err = cudaSuccess;
    for (int i = 0; i <= moe_width_index(cap) && err == cudaSuccess; ++i) {
        const cuuint64_t dim[3] = {(cuuint64_t)row_bytes, (cuuint64_t)P, kQTerms};
        const cuuint32_t box[3] = {128, (cuuint32_t)moe_width(i, cap) / 2, kQTerms};
        err = box_map(&map[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, row_bytes, base, 3, dim, box);
    }
    return err;
}
// fp16 activations [P, K]: a tile's columns, likewise
cudaError_t half_maps(CUtensorMap (&map)[kMoeWidths], const __half* base, long long P, int K, int cap) {
    cudaError_t err = cudaSuccess;
    for (int i = 0; i <= moe_width_index(cap) && err == cudaSuccess; ++i) {
        const cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)P};
        const cuuint32_t box[2] = {64, (cuuint32_t)moe_width(i, cap)};
        err = box_map(&map[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, K * 2, base, 2, dim, box);
    }
    return err;
}

// Stage timing (diagnostic; off by default): when switched on, a call records an event before its
// first kernel and after each of its stages (grouping and quantising x share a launch, and the intermediate is quantised
// inside the gate/up GEMM: those two stages read as the time between two events); mxfp4_moe_stage_times turns them into microseconds.  Events between
// the launches take away the overlap of programmatic dependent launch, so a timed call is slower than a normal one.
constexpr int kStageMarks = 7;      // start, group, quantise x, gate/up GEMM, quantise intermediate, down GEMM, combine
bool g_stage_timing = false;
cudaEvent_t g_stage_event[kStageMarks] = {};

void stage_mark(cudaStream_t stream, int i) {
    if (!g_stage_timing) return;
    if (!g_stage_event[i] && cudaEventCreate(&g_stage_event[i]) != cudaSuccess) return;
    cudaEventRecord(g_stage_event[i], stream);
}

}  // namespace

// Switches the stage timing of the block-scaled batched path on (1) or off (0); returns the previous setting.
// Not thread-safe; meant for one timed call on one stream at a time.
DSV4_API int mxfp4_moe_stage_timing(int enable) {
    const int before = g_stage_timing ? 1 : 0;
    g_stage_timing = enable != 0;
    return before;
}

// Microseconds of the six stages of the last timed call (group, quantise x, gate/up GEMM, quantise intermediate,
// down GEMM, combine) into us_out[0..6); synchronises on the last event.  Returns 0, -1 if no timed call was made.
DSV4_API int mxfp4_moe_stage_times(float* us_out) {
    if (!us_out) return -1;
    for (int i = 0; i < kStageMarks; ++i)
        if (!g_stage_event[i]) return -1;
    if (cudaEventSynchronize(g_stage_event[kStageMarks - 1]) != cudaSuccess) return -1;
    for (int i = 0; i + 1 < kStageMarks; ++i) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, g_stage_event[i], g_stage_event[i + 1]) != cudaSuccess) return -1;
        us_out[i] = ms * 1e3f;
    }
    return 0;
}

// Bytes of workspace mxfp4_moe_forward needs: grouping tables, the FP32 per-pair outputs [n_tokens * k, out_dim], and the
// activations and the intermediate of every pair in the form that needs more (three MXFP4 terms; fp16).  Three E4M3 terms of the intermediate
// lie in the same bytes, those of x in the bytes of the outputs, where there is room for them.
DSV4_API size_t mxfp4_moe_forward_workspace_bytes(int n_tokens, int k, int K_in, int hidden, int out_dim,
                                                  int n_experts) {
    if (n_tokens <= 0 || k <= 0 || K_in <= 0 || hidden <= 0 || out_dim <= 0 || n_experts <= 0) return 0;
    return map_workspace(n_tokens, k, K_in, hidden, out_dim, n_experts).total;
}

// x bf16 [n_tokens, K_in]; bank tensors stacked over n_experts as in mxfp4_grouped_gemv_topk_ids; ids int32
// [n_tokens, k] (a token lists an expert at most once; a negative id marks a pair to skip, which is how an
// expert-parallel caller masks the experts of other ranks), weights FP32 [n_tokens, k]; out bf16 [n_tokens, out_dim].
// Shapes: K_in and hidden multiples of 256, hidden and out_dim multiples of 128, n_experts <= 1024.
// Returns 0, -1 bad shape, -2 null / misaligned pointer, -3 launch failure.
static int moe_forward_impl(int path, const __nv_bfloat16* x, const uint8_t* bank_W1_packed, const uint8_t* bank_W3_packed,
                               const uint8_t* bank_W2_packed, const uint8_t* bank_W1_scale,
                               const uint8_t* bank_W3_scale, const uint8_t* bank_W2_scale, const int* ids,
                               const float* weights, int n_tokens, int n_experts, int K_in, int hidden, int out_dim,
                               int k, __nv_bfloat16* out, void* workspace, cudaStream_t stream,
                               const MoePeerOut* peer = nullptr, const MoePeerIn* peer_in = nullptr) {
    const char* who = "mxfp4_moe_forward";
    if (path != 0 && path != 1) return -1;
    if (n_tokens < 0 || k <= 0 || n_experts <= 0 || n_experts > kMoeMaxExperts || K_in <= 0 || K_in % 256 != 0 ||
        hidden <= 0 || hidden % 256 != 0 || out_dim <= 0 || out_dim % 128 != 0 || K_in > 16384 || hidden > 16384) {
        std::fprintf(stderr, "%s: unsupported shape T=%d E=%d K=%d H=%d O=%d k=%d\n", who, n_tokens, n_experts, K_in,
                     hidden, out_dim, k);
        return -1;
    }
    if (n_tokens == 0) return 0;
    if ((!x && !peer_in) || !bank_W1_packed || !bank_W3_packed || !bank_W2_packed || !bank_W1_scale || !bank_W3_scale ||
        !bank_W2_scale || !ids || !weights || (!out && !peer) || !workspace || (x && !aligned16(x)) || !aligned16(bank_W1_packed) ||
        !aligned16(bank_W3_packed) || !aligned16(bank_W2_packed) || !aligned16(bank_W1_scale) ||
        !aligned16(bank_W3_scale) || !aligned16(bank_W2_scale) || !aligned16(workspace) || (out && !aligned16(out))) {
        std::fprintf(stderr, "%s: null pointer or a tensor that is not 16-byte aligned\n", who);
        return -2;
    }
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    const WorkspaceMap m = map_workspace(n_tokens, k, K_in, hidden, out_dim, n_experts);
    const int P = n_tokens * k;
    MoeGroups g;
    g.offsets = reinterpret_cast<int*>(ws + m.offsets);
    g.tiles_up = reinterpret_cast<int*>(ws + m.tiles_up);
    g.tiles_down = reinterpret_cast<int*>(ws + m.tiles_down);
    g.pair_slot = reinterpret_cast<int*>(ws + m.pair_slot);
    g.slot_w = reinterpret_cast<float*>(ws + m.slot_w);
    float* y = reinterpret_cast<float*>(ws + m.y);

    int* status = nullptr;
    cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_device_status);
    stage_mark(stream, 0);
    const int grid = sm_count();

    MoeGroupArgs ga;
    ga.ids = ids; ga.weights = weights; ga.n_pairs = P; ga.n_experts = n_experts; ga.g = g; ga.status = status;
    // Path 0 runs on the block-scaled MMAs too, with E4M3 terms, where its operands have room and the TMA can lay the weights down.
    auto aligned32 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; };
    const bool fp8 = path == 0 && !peer_in && m.fits8 && P <= (long long)kQMostTokensFp8 * n_experts && aligned32(bank_W1_packed) &&
                     aligned32(bank_W3_packed) && aligned32(bank_W2_packed);
    const bool pairs = path == 1 || fp8;                   // tiles of CTA pairs
    const int rows_up = pairs ? kQTileRowsUp : kMoeTileRows, rows_down = pairs ? kQTileRowsDown : 2 * kMoeTileRows;
    ga.m_tiles_up = hidden / rows_up; ga.m_tiles_down = (out_dim + rows_down - 1) / rows_down;
    // (Pairs of the whole batch: where ids are negative, as under expert parallelism, the experts here have fewer.  Eight ranks emulated on
    // one GPU, 32 experts of 4096, 2048 each, top 6: the larger tiles although the smaller would do cost 1 % of the layer's time from 128 to 1024
    // tokens; fp16 MMAs although E4M3 terms would do, path 0, 512 tokens 178 us where 144 would do, 1 024 194 / 156, 2 048 222 / 184.)
    const int cap16 = P <= (long long)kTmFewTokens * n_experts ? 64 : kMoeTileTokens;      // tokens per tile, fp16 path
    const bool few = P <= (long long)(fp8 ? kQFewTokensFp8 : kQFewTokens) * n_experts;
    const int cap_q = few ? 32 : kQTok;                                                    // tokens per tile, block-scaled path
    ga.tile_tokens = pairs ? cap_q : cap16;
    ga.typical.w1_s = bank_W1_scale; ga.typical.w3_s = bank_W3_scale; ga.typical.K = K_in; ga.typical.hidden = hidden;
    ga.typical.n_experts = n_experts; ga.typical.typical = reinterpret_cast<int*>(ws + (fp8 ? m.typical8 : m.typical));
    ga.blocks = P > kGroupOneBlockPairs ? kGroupCluster : 1;
    // E4M3 terms: further blocks of the grouping kernel look for the typical scales (fp16 MMAs: blocks of the activation kernel do)
    const int scale_blocks = (n_experts + kTypicalExperts - 1) / kTypicalExperts;
    const int ggrid = ga.blocks + (fp8 ? (scale_blocks + ga.blocks - 1) / ga.blocks * ga.blocks : 0);
    launch_k(moe_group_kernel, dim3(ggrid), dim3(kPrepThreads), 0, stream, ga.blocks, ga);
    stage_mark(stream, 1);

    MoeActArgs aa;
    aa.x = x; aa.pair_slot = g.pair_slot; aa.n_tokens = n_tokens; aa.k = k; aa.K = K_in; aa.n_pairs = P;
    aa.q = ws + m.xq; aa.s = ws + m.xs; aa.xh = reinterpret_cast<__half*>(ws + m.xh);
    aa.xexp = reinterpret_cast<int2*>(ws + m.xexp); aa.ids = ids; aa.row_exp = reinterpret_cast<int*>(ws + m.row_exp8);
    aa.typical = ga.typical;
    const MoePeerIn no_peers = {};
    const MoePeerIn& pin = peer_in ? *peer_in : no_peers;
    cudaError_t err = cudaSuccess;
    if (pairs) {
        // ---- block-scaled MMAs.  MXFP4 terms of x: a warp per 256 elements, at most eight blocks of eight warps per SM; where that
        // fills the SMs, a warp per 1024, two blocks.  E4M3 terms: blocks of whole rows, as many as the registers of an SM hold.
        const bool many = !peer_in && moe_act_by_blocks(n_tokens, K_in);
        const long long pieces = (long long)n_tokens * (many ? (K_in + 1023) / 1024 : K_in / 256);
        const int act8_rows = kAct8Warps / moe_act8_row_warps(K_in), act8_pieces = (K_in + 512 * kAct8Warps - 1) / (512 * kAct8Warps);
        const long long blocks = fp8 ? (n_tokens + act8_rows - 1) / act8_rows : (pieces + 7) / 8;
        const long long most = (fp8 ? (act8_pieces == 1 ? 4LL : act8_pieces == 2 ? 3LL : 2LL) : many ? 2LL : 8LL) * grid;
        uint8_t* const mid_q = ws + (fp8 ? m.mq8 : m.mq);
        uint8_t* const mid_s = ws + (fp8 ? m.ms8 : m.ms);
        if (fp8) { aa.q = ws + m.xq8; aa.s = ws + m.xs8; }
        const dim3 agrid((unsigned)(blocks < most ? blocks : most)), ablock(256);
        if (fp8)
            launch_k(act8_pieces == 1 ? moe_act_fp8_kernel<1> : act8_pieces == 2 ? moe_act_fp8_kernel<2> : moe_act_fp8_kernel<4>, agrid,
                     ablock, 0, stream, 1, aa);
        else if (many) launch_k(moe_act_blocks_kernel, agrid, ablock, 0, stream, 1, aa);
        else launch_k(peer_in ? moe_act_mxf4_kernel<true> : moe_act_mxf4_kernel<false>, agrid, ablock, 0, stream, 1, aa, pin);
        stage_mark(stream, 2);
        MoeQMaps up_maps, down_maps;
        auto weights = [&](CUtensorMap* map, const uint8_t* base, long long rows, int K) {
            if (err == cudaSuccess) err = fp8 ? weight_map_padded(map, base, rows, K) : weight_map(map, base, rows, K);
        };
        weights(&up_maps.wa, bank_W1_packed, (long long)n_experts * hidden, K_in);
        weights(&up_maps.wb, bank_W3_packed, (long long)n_experts * hidden, K_in);
        weights(&down_maps.wa, bank_W2_packed, (long long)n_experts * out_dim, hidden);
        down_maps.wb = down_maps.wa;
        if (err == cudaSuccess) err = term_maps(up_maps.act, aa.q, P, fp8 ? K_in : K_in / 2, cap_q);
        if (err == cudaSuccess) err = term_maps(down_maps.act, mid_q, P, fp8 ? hidden : hidden / 2, cap_q);
        MoeQGemmArgs qu;
        qu.wa_s = bank_W1_scale; qu.wb_s = bank_W3_scale; qu.rows = hidden; qu.K = K_in; qu.n_experts = n_experts;
        qu.act_s = aa.s; qu.row_exp = aa.row_exp; qu.n_pairs = P; qu.g = g; qu.mid_q = mid_q; qu.mid_s = mid_s; qu.y = nullptr;
        MoeQGemmArgs qd = qu;
        qd.wa_s = bank_W2_scale; qd.wb_s = nullptr; qd.rows = out_dim; qd.K = hidden; qd.act_s = mid_s; qd.y = y;
        auto gemms = [&](auto format, auto cap) {
            using F = decltype(format);
            constexpr int CAP = decltype(cap)::value;
            auto up_kernel = moe_gemm_mxf4_kernel<0, CAP, F>;
            auto down_kernel = moe_gemm_mxf4_kernel<1, CAP, F>;
            static int up_done[64] = {0}, down_done[64] = {0};
            const uint32_t smem = MoeQShape<F, CAP>::smem(n_experts), most_smem = MoeQShape<F, CAP>::smem(kMoeMaxExperts);
            if (err == cudaSuccess) err = allow_smem(up_kernel, most_smem, up_done);
            if (err == cudaSuccess) err = allow_smem(down_kernel, most_smem, down_done);
            if (err != cudaSuccess) return;
            launch_k(up_kernel, dim3(grid & ~1), dim3(kQThreads), smem, stream, 2, up_maps, qu);
            stage_mark(stream, 3);
            stage_mark(stream, 4);
            launch_k(down_kernel, dim3(grid & ~1), dim3(kQThreads), smem, stream, 2, down_maps, qd);
        };
        const std::integral_constant<int, 32> cap_few;
        const std::integral_constant<int, kQTok> cap_most;
        if (fp8) { if (few) gemms(MoeQFp8(), cap_few); else gemms(MoeQFp8(), cap_most); }
        else if (few) gemms(MoeQFp4(), cap_few);
        else gemms(MoeQFp4(), cap_most);
    } else {
        // ---- fp16 tensor-core path: weights dequantised into tensor memory
        const int blocks = (n_tokens + kActRows - 1) / kActRows;
        const dim3 agrid(scale_blocks + (blocks < 2 * grid ? blocks : 2 * grid)), ablock(kPrepThreads);
        launch_k(peer_in ? moe_act_fp16_kernel<true> : moe_act_fp16_kernel<false>, agrid, ablock, 0, stream, 1, aa, pin);
        stage_mark(stream, 2);
        __half* mid = reinterpret_cast<__half*>(ws + m.mid);
        MoeMaps up_maps, down_maps;
        err = weight_map(&up_maps.wa, bank_W1_packed, (long long)n_experts * hidden, K_in);
        if (err == cudaSuccess) err = weight_map(&up_maps.wb, bank_W3_packed, (long long)n_experts * hidden, K_in);
        if (err == cudaSuccess) err = half_maps(up_maps.act, aa.xh, P, K_in, cap16);
        if (err == cudaSuccess) err = weight_map(&down_maps.wa, bank_W2_packed, (long long)n_experts * out_dim, hidden);
        down_maps.wb = down_maps.wa;
        if (err == cudaSuccess) err = half_maps(down_maps.act, mid, P, hidden, cap16);
        MoeGemmArgs up;
        up.wa_s = bank_W1_scale; up.wb_s = bank_W3_scale; up.rows = hidden; up.K = K_in; up.n_experts = n_experts;
        up.xexp = aa.xexp; up.typical = aa.typical.typical; up.g = g;
        up.mid_log = 2;
        while ((2 << (up.mid_log - 2)) <= K_in) ++up.mid_log;                // floor(log2(K)) + 2
        up.mid = mid; up.mid_exp = reinterpret_cast<int*>(ws + m.mid_exp); up.y = y;
        MoeGemmArgs down = up;
        down.wa_s = bank_W2_scale; down.wb_s = nullptr; down.rows = out_dim; down.K = hidden;
        auto gemms = [&](auto up_kernel, auto down_kernel, uint32_t smem, int (&up_done)[64], int (&down_done)[64]) {
            if (err == cudaSuccess) err = allow_smem(up_kernel, smem, up_done);
            if (err == cudaSuccess) err = allow_smem(down_kernel, smem, down_done);
            if (err != cudaSuccess) return;
            launch_k(up_kernel, dim3(grid), dim3(kTmThreads), smem, stream, 1, up_maps, up);
            stage_mark(stream, 3);
            stage_mark(stream, 4);
            launch_k(down_kernel, dim3(grid), dim3(kTmThreads), smem, stream, 1, down_maps, down);
        };
        static int up64[64] = {0}, down64[64] = {0}, up128[64] = {0}, down128[64] = {0};
        if (cap16 == 64) gemms(moe_gemm_kernel<0, 64>, moe_gemm_kernel<1, 64>, MoeTmShape<64>::kSmem, up64, down64);
        else gemms(moe_gemm_kernel<0, 128>, moe_gemm_kernel<1, 128>, MoeTmShape<128>::kSmem, up128, down128);
    }
    if (err == cudaSuccess) {
        stage_mark(stream, 5);
        dim3 cgrid((out_dim / 4 + 127) / 128, n_tokens < 65535 ? n_tokens : 65535);
        if (peer)
            launch_k(moe_combine_peer_kernel, dim3(cgrid), dim3(128), 0, stream, 1, y, g.pair_slot, n_tokens, k, out_dim, *peer);
        else
            launch_k(moe_combine_kernel, dim3(cgrid), dim3(128), 0, stream, 1, y, g.pair_slot, n_tokens, k, out_dim, out);
        stage_mark(stream, 6);
        err = cudaGetLastError();
    }
    if (err != cudaSuccess) {
        std::fprintf(stderr, "%s: launch failed: %s\n", who, cudaGetErrorString(err));
        return -3;
    }
    return 0;
}

// The tensor-core path of the entries that leave it to the library: block-scaled MXFP4 MMAs; DSV4_B200_MOE_PATH=fp16 in
// the environment selects the fp16 path.
static int default_path() {
    static int path = -1;
    if (path < 0) {
        const char* e = std::getenv("DSV4_B200_MOE_PATH");
        path = (e && e[0] == 'f') ? 0 : 1;
    }
    return path;
}

DSV4_API int mxfp4_moe_forward(const __nv_bfloat16* x, const uint8_t* bank_W1_packed, const uint8_t* bank_W3_packed,
                               const uint8_t* bank_W2_packed, const uint8_t* bank_W1_scale,
                               const uint8_t* bank_W3_scale, const uint8_t* bank_W2_scale, const int* ids,
                               const float* weights, int n_tokens, int n_experts, int K_in, int hidden, int out_dim,
                               int k, __nv_bfloat16* out, void* workspace, cudaStream_t stream) {
    return moe_forward_impl(default_path(), x, bank_W1_packed, bank_W3_packed, bank_W2_packed, bank_W1_scale, bank_W3_scale,
                            bank_W2_scale, ids, weights, n_tokens, n_experts, K_in, hidden, out_dim, k, out, workspace,
                            stream);
}

// The same with the tensor-core path chosen by the caller: 0 = "fp16" (moe_gemm.cuh says what its two forms
// hold exactly), 1 = block-scaled MXFP4 MMAs (weights as stored, activations as three MXFP4 terms).
DSV4_API int mxfp4_moe_forward_path(int path, const __nv_bfloat16* x, const uint8_t* bank_W1_packed,
                                    const uint8_t* bank_W3_packed, const uint8_t* bank_W2_packed,
                                    const uint8_t* bank_W1_scale, const uint8_t* bank_W3_scale,
                                    const uint8_t* bank_W2_scale, const int* ids, const float* weights, int n_tokens,
                                    int n_experts, int K_in, int hidden, int out_dim, int k, __nv_bfloat16* out,
                                    void* workspace, cudaStream_t stream) {
    return moe_forward_impl(path, x, bank_W1_packed, bank_W3_packed, bank_W2_packed, bank_W1_scale, bank_W3_scale,
                            bank_W2_scale, ids, weights, n_tokens, n_experts, K_in, hidden, out_dim, k, out, workspace,
                            stream);
}

// 0 unless a kernel of this library gave up on a bounded wait (4 producer, 5 MMA issuer, 6 epilogue) or met an
// expert id outside the bank (3) since the last call; clears the status.  Synchronises the device.
DSV4_API int mxfp4_moe_device_status(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_device_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int));
    return v;
}

// Expert parallel, combine fused with the exchange: the layer of mxfp4_moe_forward over the GATHERED batch of
// world * tokens_per_rank tokens (token t belongs to rank t / tokens_per_rank; ids index this rank's local bank, -1
// where the expert lives elsewhere), whose per-token sums are not written to a local output but stored by the
// combine kernel straight into the receive buffer of the token's home rank - peer memory, plain stores over NVLink,
// the transfer being the kernel's own epilogue.  recv_ptrs: HOST array of `world` device pointers, entry r the
// receive buffer of rank r, bf16 [world][tokens_per_rank][out_dim] (peer-mapped, e.g. symmetric memory); this rank
// writes slice [my_rank] of each.  After a barrier over the ranks every rank calls mxfp4_moe_ep_sum on its own
// buffer.  Return codes as mxfp4_moe_forward; -1 also for world outside 1..16 or a token count that is not
// world * tokens_per_rank.
DSV4_API int mxfp4_moe_forward_ep(const __nv_bfloat16* x, const uint8_t* bank_W1_packed, const uint8_t* bank_W3_packed,
                                  const uint8_t* bank_W2_packed, const uint8_t* bank_W1_scale,
                                  const uint8_t* bank_W3_scale, const uint8_t* bank_W2_scale, const int* ids,
                                  const float* weights, int n_tokens, int n_experts, int K_in, int hidden, int out_dim,
                                  int k, void* const* recv_ptrs, int world, int my_rank, int tokens_per_rank,
                                  void* workspace, cudaStream_t stream) {
    if (world < 1 || world > kMoeMaxRanks || my_rank < 0 || my_rank >= world || tokens_per_rank <= 0 ||
        n_tokens != world * tokens_per_rank || !recv_ptrs) {
        std::fprintf(stderr, "mxfp4_moe_forward_ep: bad rank layout world=%d rank=%d tokens_per_rank=%d n_tokens=%d\n", world,
                     my_rank, tokens_per_rank, n_tokens);
        return -1;
    }
    MoePeerOut peer = {};
    for (int r = 0; r < world; ++r) {
        if (!recv_ptrs[r] || !aligned16(recv_ptrs[r])) return -2;
        peer.recv[r] = reinterpret_cast<__nv_bfloat16*>(recv_ptrs[r]);
    }
    peer.world = world; peer.my_rank = my_rank; peer.tokens_per_rank = tokens_per_rank;
    return moe_forward_impl(default_path(), x, bank_W1_packed, bank_W3_packed, bank_W2_packed, bank_W1_scale, bank_W3_scale,
                            bank_W2_scale, ids, weights, n_tokens, n_experts, K_in, hidden, out_dim, k, nullptr,
                            workspace, stream, &peer);
}

// out[t] = bf16(sum of recv[r][t] over the ranks r that own one of token t's experts, in ascending order): the home
// rank's side of mxfp4_moe_forward_ep, after the barrier.  recv bf16 [world][n_tokens][out_dim]; ids int32
// [n_tokens, k] GLOBAL expert ids of this rank's tokens (a rank owns experts [r, r + 1) * experts_per_rank; ranks
// without an expert of the token stored nothing and are skipped); out bf16 [n_tokens][out_dim]; out_dim a multiple
// of 4, world <= 16.  Returns 0, -1 bad shape, -2 null / misaligned pointer, -3 launch failure.
DSV4_API int mxfp4_moe_ep_sum(const __nv_bfloat16* recv, const int* ids, int k, int experts_per_rank, int world,
                              int n_tokens, int out_dim, __nv_bfloat16* out, cudaStream_t stream) {
    if (world < 1 || world > kMoeMaxRanks || n_tokens < 0 || out_dim <= 0 || out_dim % 4 != 0 || k <= 0 ||
        experts_per_rank <= 0)
        return -1;
    if (n_tokens == 0) return 0;
    if (!recv || !ids || !out || !aligned16(recv) || !aligned16(out)) return -2;
    const long long n4 = (long long)n_tokens * out_dim / 4;
    long long grid = (n4 + 255) / 256;
    if (grid > 8LL * sm_count()) grid = 8LL * sm_count();
    launch_k(moe_ep_sum_kernel, dim3((unsigned)grid), dim3(256), 0, stream, 1, recv, ids, k, experts_per_rank, world,
             n_tokens, out_dim, out);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// Expert parallel with BOTH sides over peer memory (no collective library on the path): every rank publishes its
// tokens in buffers that are mapped on all ranks (symmetric memory): x bf16 [tokens_per_rank, K_in], ids int32
// [tokens_per_rank, k] (global expert ids), weights FP32 [tokens_per_rank, k].  After a barrier over the ranks this
// call runs the rank's experts over the whole batch of world * tokens_per_rank tokens: a small kernel turns the
// published ids into this rank's view (local index, -1 for experts of other ranks), the activation quantiser reads
// every token's row from the rank that published it (plain loads over NVLink), and the combine kernel stores the
// partial rows into the home ranks' receive buffers as in mxfp4_moe_forward_ep.  x_ptrs / ids_ptrs / w_ptrs /
// recv_ptrs: HOST arrays of `world` device pointers.  workspace:
// mxfp4_moe_forward_ep2_workspace_bytes.  Return codes as mxfp4_moe_forward_ep.
DSV4_API size_t mxfp4_moe_forward_ep2_workspace_bytes(int world, int tokens_per_rank, int k, int K_in, int hidden,
                                                      int out_dim, int n_experts_local) {
    if (world <= 0 || tokens_per_rank <= 0 || k <= 0) return 0;
    const long long T = (long long)world * tokens_per_rank;
    const size_t base = map_workspace(T, k, K_in, hidden, out_dim, n_experts_local).total;
    return base + 2 * (((size_t)T * k * 4 + 255) & ~size_t(255));
}

DSV4_API int mxfp4_moe_forward_ep2(void* const* x_ptrs, void* const* ids_ptrs, void* const* w_ptrs,
                                   const uint8_t* bank_W1_packed, const uint8_t* bank_W3_packed,
                                   const uint8_t* bank_W2_packed, const uint8_t* bank_W1_scale,
                                   const uint8_t* bank_W3_scale, const uint8_t* bank_W2_scale, int tokens_per_rank,
                                   int n_experts_local, int K_in, int hidden, int out_dim, int k,
                                   void* const* recv_ptrs, int world, int my_rank, void* workspace,
                                   cudaStream_t stream) {
    if (world < 1 || world > kMoeMaxRanks || my_rank < 0 || my_rank >= world || tokens_per_rank <= 0 || k <= 0 ||
        n_experts_local <= 0 || !x_ptrs || !ids_ptrs || !w_ptrs || !recv_ptrs || !workspace) {
        std::fprintf(stderr, "mxfp4_moe_forward_ep2: bad rank layout or null table\n");
        return -1;
    }
    MoePeerIn in = {};
    MoePeerOut peer = {};
    for (int r = 0; r < world; ++r) {
        if (!x_ptrs[r] || !ids_ptrs[r] || !w_ptrs[r] || !recv_ptrs[r] || !aligned16(x_ptrs[r]) || !aligned16(recv_ptrs[r]))
            return -2;
        in.x[r] = reinterpret_cast<const __nv_bfloat16*>(x_ptrs[r]);
        in.ids[r] = reinterpret_cast<const int*>(ids_ptrs[r]);
        in.w[r] = reinterpret_cast<const float*>(w_ptrs[r]);
        peer.recv[r] = reinterpret_cast<__nv_bfloat16*>(recv_ptrs[r]);
    }
    in.world = peer.world = world; in.my_rank = peer.my_rank = my_rank;
    in.tokens_per_rank = peer.tokens_per_rank = tokens_per_rank; in.experts_per_rank = n_experts_local;
    const int n_tokens = world * tokens_per_rank;
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    const size_t base = map_workspace(n_tokens, k, K_in, hidden, out_dim, n_experts_local).total;
    int* ids_local = reinterpret_cast<int*>(ws + base);
    float* w_local = reinterpret_cast<float*>(ws + base + (((size_t)n_tokens * k * 4 + 255) & ~size_t(255)));
    const int n_meta = n_tokens * k;
    launch_k(moe_ep_gather_meta_kernel, dim3((unsigned)((n_meta + 255) / 256)), dim3(256), 0, stream, 1, in, k, ids_local,
             w_local);
    return moe_forward_impl(default_path(), nullptr, bank_W1_packed, bank_W3_packed, bank_W2_packed, bank_W1_scale, bank_W3_scale,
                            bank_W2_scale, ids_local, w_local, n_tokens, n_experts_local, K_in, hidden, out_dim, k,
                            nullptr, workspace, stream, &peer, &in);
}

// Tensor-pipe clocks of one tcgen05.mma kind::mxf4 (M = 128, K = 64, N = n_cols: a multiple of 16 in 16 .. 256) with
// `scale_copies` (0 .. 8) scale-atom copies issued in front of every four MMAs; one CTA per SM, `iters` rounds of
// four MMAs.  clocks_per_mma: HOST pointer.  `scratch`: 8 bytes of device memory.  Synchronises the stream.
// Returns 0, -1 bad argument, -3 launch / execution failure.
DSV4_API int mxfp4_moe_mma_rate(int n_cols, int scale_copies, int iters, void* scratch, double* clocks_per_mma,
                                cudaStream_t stream) {
    if (n_cols < 16 || n_cols > 256 || n_cols % 16 != 0 || scale_copies < 0 || scale_copies > 8 || iters <= 0 ||
        iters > (1 << 20) || !scratch || !clocks_per_mma)
        return -1;
    static int done[64] = {0};
    if (allow_smem(mxf4_mma_rate_kernel, kRateBytes, done) != cudaSuccess) return -3;
    long long* dev_clocks = reinterpret_cast<long long*>(scratch);
    mxf4_mma_rate_kernel<<<sm_count(), 128, kRateBytes, stream>>>(n_cols, 8, scale_copies, dev_clocks);       // warm-up
    mxf4_mma_rate_kernel<<<sm_count(), 128, kRateBytes, stream>>>(n_cols, iters, scale_copies, dev_clocks);
    long long clocks = 0;
    if (cudaMemcpyAsync(&clocks, dev_clocks, sizeof(clocks), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return -3;
    *clocks_per_mma = (double)clocks / (4.0 * iters);
    return 0;
}
