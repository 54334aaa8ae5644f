// MUL_MAT over Q4_K / Q6_K weights for 1..16 activation rows, and the Q8_K
// activation quantiser.  Replaces cb_gemv_custom / cb_gemv_batched_custom
// (core/src/llm/matmul/gemv_exec.cpp:99, core/src/llm/matmul/batched_exec.cpp:55).
//
// Weights stay in their GGUF-native 144-byte / 210-byte super-blocks; dc_rows.cuh
// holds the kernel's body.
#include <stdarg.h>
#include <stdio.h>

#include "dc_common.cuh"
#include "dc_internal.h"
#include "dc_launch.cuh"
#include "dc_rows.cuh"

using namespace dc;

template <bool FRAG>
__global__ void __launch_bounds__(256) k_quantize_q8k(const float* __restrict__ x, int n_blocks,
                                                      uint8_t* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int b = gw; b < n_blocks; b += nw)
        quantize_block_q8k_warp<FRAG>(x + (size_t)b * DC_QK_K, out + (size_t)b * (FRAG ? DC_Q8F_BYTES : DC_Q8K_BYTES), lane);
}

int dc_launch_quantize_q8k(dc_ctx* ctx, const float* x, int rows, int K, uint8_t* out, bool frag) {
    const int n_blocks = rows * (K / DC_QK_K);
    const int grid = (n_blocks + 7) / 8;
    (frag ? k_quantize_q8k<true> : k_quantize_q8k<false>)<<<grid < 1 ? 1 : grid, 256, 0, ctx->stream>>>(x, n_blocks, out);
    return dc_check_cuda(ctx, cudaGetLastError(), "k_quantize_q8k");
}

// ------------------------------------------------------------------- rows
// KIND: matrices of Q4_K, of Q6_K, or of both, where every CTA works on one type.  Weights do not depend on the previous kernel:
// they stream in while this one waits for it.
enum { ROWS_Q4K = 0, ROWS_Q6K = 1, ROWS_BOTH = 2 };
template <int KIND, int NP, bool ONE, bool ALONE, bool PAIR, bool DUMP>
__global__ void __launch_bounds__(RW_THREADS, NP > 4 ? 1 : KIND == ROWS_Q4K ? 3 : 2) k_rows(const RowsParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    if (KIND == ROWS_Q4K || (KIND == ROWS_BOTH && blockIdx.x < p.ctas4)) {
        rows_cta<DC_TYPE_Q4_K, NP, ONE, ALONE, false, PAIR, DUMP, true>(p, smem, blockIdx.x, p.ctas4, 0, p.tiles4);
    } else {
        rows_cta<DC_TYPE_Q6_K, NP, ONE, ALONE, false, PAIR, DUMP, true>(p, smem, blockIdx.x - p.ctas4, gridDim.x - p.ctas4, p.tiles4, p.tiles);
    }
}

template <int KIND, int NP, bool ONE, bool PAIR, bool DUMP, bool ALONE>
static int launch_rows_as(dc_ctx* ctx, RowsParams& p, size_t smem) {
    const void* f = (const void*)k_rows<KIND, NP, ONE, ALONE, PAIR, DUMP>;
    int st = dc_kernel_setup(ctx, f, 220 * 1024, "cudaFuncSetAttribute(k_rows)");
    if (st != DC_B200_OK) return st;
    int per_sm = dc_kernel_occupancy(ctx, f, RW_THREADS, smem);
    if (per_sm < 1) per_sm = 1;
    const int groups = RW_WARPS / p.S, slots = ctx->num_sms * per_sm;
    const int n4 = (p.tiles4 + groups - 1) / groups, n6 = (p.tiles - p.tiles4 + groups - 1) / groups;
    int c4 = n4, c6 = n6;
    if (c4 + c6 > slots) {     // shared out by cost: a Q6_K tile takes about twice the instructions of a Q4_K tile
        c6 = n6 ? (int)(2ll * n6 * slots / (n4 + 2ll * n6)) : 0;
        if (n6 && c6 < 1) c6 = 1;
        c4 = n4 ? (slots - c6 < 1 ? 1 : slots - c6) : 0;
        if (c6 > n6) c6 = n6;
        if (c4 > n4) c4 = n4;
    }
    p.ctas4 = c4;
    return dc_launch(ctx, "k_rows", k_rows<KIND, NP, ONE, ALONE, PAIR, DUMP>, dim3(c4 + c6), dim3(RW_THREADS), smem, p);
}
template <int KIND, int NP, bool ONE, bool PAIR, bool DUMP>
static int launch_rows(dc_ctx* ctx, RowsParams& p, size_t smem) {
    return p.S == 1 ? launch_rows_as<KIND, NP, ONE, PAIR, DUMP, true>(ctx, p, smem) : launch_rows_as<KIND, NP, ONE, PAIR, DUMP, false>(ctx, p, smem);
}
template <int KIND, bool PAIR, bool DUMP = false>
static int launch_rows_np(dc_ctx* ctx, RowsParams& p, int np, size_t smem) {
    if (p.T == 1) return launch_rows<KIND, 1, true, PAIR, DUMP>(ctx, p, smem);
    if (np == 1) return launch_rows<KIND, 1, false, PAIR, DUMP>(ctx, p, smem);
    if (np == 2) return launch_rows<KIND, 2, false, PAIR, DUMP>(ctx, p, smem);
    if (np == 4) return launch_rows<KIND, 4, false, PAIR, DUMP>(ctx, p, smem);
    return launch_rows<KIND, 8, false, PAIR, DUMP>(ctx, p, smem);
}

int dc_launch_gemv(dc_ctx* ctx, const dc_gemv_seg* segs, int n_seg, int epi, const uint8_t* act_q8, int T, int K,
                   unsigned long long* argmax, int32_t* dump_I, int32_t* dump_M, const float* act_f32, const float* norm_w, float norm_eps) {
    if (n_seg < 1 || n_seg > 3 || T < 1 || T > DC_MAX_T || K % DC_QK_K)
        return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemv: bad shape (n_seg=%d T=%d K=%d)", n_seg, T, K);
    RowsParams p = {};
    p.n_seg = epi == DC_EPI_SWIGLU ? 1 : n_seg;
    p.epi = epi;
    p.act_q8 = act_q8;
    p.act_f32 = act_f32;
    p.norm_w = act_f32 ? norm_w : nullptr;
    if (p.norm_w && !dc_rows_quantise(T, K)) return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemv: too many rows to norm (T=%d K=%d)", T, K);
    p.norm_eps = norm_eps;
    p.T = p.act_rows = T;
    p.K = K;
    p.nb = K / DC_QK_K;
    p.argmax = argmax;
    if (dump_I) {
        if (n_seg != 1 || epi != DC_EPI_STORE) return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemv: block-sum capture takes one plain segment");
        p.dump = BlockSumDump{dump_I, dump_M, segs[0].n_rows};
    }
    if (epi == DC_EPI_SWIGLU && (n_seg != 2 || segs[0].n_rows != segs[1].n_rows || segs[0].type != segs[1].type))
        return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemv: SwiGLU needs matching gate/up segments");
    bool q4 = false, q6 = false;
    for (int i = 0; i < n_seg; ++i) {
        if (segs[i].type != DC_TYPE_Q4_K && segs[i].type != DC_TYPE_Q6_K)
            return dc_fail(ctx, DC_B200_UNSUPPORTED, "gemv: weight type %d is not Q4_K/Q6_K", segs[i].type);
        (segs[i].type == DC_TYPE_Q4_K ? q4 : q6) = true;
    }
    int n = 0;
    for (int type : {DC_TYPE_Q4_K, DC_TYPE_Q6_K}) {
        for (int i = 0; i < n_seg; ++i) {
            if (segs[i].type != type) continue;
            p.seg[n] = segs[i];
            if (n < p.n_seg) p.tiles += p.seg_tiles[n] = (segs[i].n_rows + 15) / 16;
            ++n;
        }
        if (type == DC_TYPE_Q4_K) p.tiles4 = p.tiles;
    }
    const bool pair = epi == DC_EPI_SWIGLU;
    const int np = T <= 2 ? 1 : T <= 4 ? 2 : T <= 8 ? 4 : 8;
    const size_t smem = rows_plan(p, np, q6, p.tiles, ctx->num_sms);
    if (!smem) {
        // activations of all T tokens do not fit beside the weight pipeline: run the tokens in two halves
        if (T == 1 || argmax || dump_I) return dc_fail(ctx, DC_B200_UNSUPPORTED, "gemv: K=%d needs too much shared memory for %d tokens", K, T);
        const int T0 = T / 2;
        dc_gemv_seg second[3];
        for (int i = 0; i < n_seg; ++i) {
            second[i] = segs[i];
            second[i].out = segs[i].out + (size_t)T0 * segs[i].ldo;
        }
        int st = dc_launch_gemv(ctx, segs, n_seg, epi, act_q8, T0, K, nullptr, nullptr, nullptr, act_f32, norm_w, norm_eps);
        if (st != DC_B200_OK) return st;
        return dc_launch_gemv(ctx, second, n_seg, epi, act_q8 + (size_t)T0 * (K / DC_QK_K) * DC_Q8F_BYTES, T - T0, K, nullptr, nullptr, nullptr,
                              act_f32 ? act_f32 + (size_t)T0 * K : nullptr, norm_w, norm_eps);
    }
    // parity capture of the block sums: the instance that serves so many tokens, compiled with the stores in (never in a decoder step)
    if (dump_I) return q4 ? launch_rows_np<ROWS_Q4K, false, true>(ctx, p, np, smem) : launch_rows_np<ROWS_Q6K, false, true>(ctx, p, np, smem);
    if (pair) return q4 ? launch_rows_np<ROWS_Q4K, true>(ctx, p, np, smem) : launch_rows_np<ROWS_Q6K, true>(ctx, p, np, smem);
    if (q4 && q6) return launch_rows_np<ROWS_BOTH, false>(ctx, p, np, smem);
    return q4 ? launch_rows_np<ROWS_Q4K, false>(ctx, p, np, smem) : launch_rows_np<ROWS_Q6K, false>(ctx, p, np, smem);
}
