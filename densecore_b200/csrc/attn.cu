// Paged-KV split-K flash-decode attention.  Replaces cb_paged_attention_decode
// (core/src/llm/attention/paged_exec.cpp:343) and its kernel PagedAttentionImpl
// (core/src/kernels/hwy/hwy_paged_attention.cc:367-630).
//
// The reference walks a sequence's 16-token KV blocks in order with an online
// softmax: m_b = max(m_{b-1}, block max), alpha_b = fastexp(m_{b-1} - m_b),
// acc = acc*alpha_b + sum_t fastexp(s_t - m_b) v_t, and finally acc/(d + 1e-6).
// fastexp is a cubic polynomial, so the result depends on which maximum each
// exponent is taken against.  To stay on the reference's numbers while cutting
// the sequence into parallel runs, a cluster of CTAs shares it (k_attn_cluster,
// below) where that is the faster form and its keys fit into the cluster's shared memory; else two kernels do it:
//   k_attn_scores  every run computes its scores s_t and per-block maxima;
//   k_attn_pv      every run rebuilds the reference's running-maximum chain from
//                  ALL block maxima (so its exponents are taken against exactly
//                  the reference's m_b), accumulates its blocks as the reference
//                  does, scales its partial by the product of the alphas of all
//                  later blocks, and the last run to finish (a ticket, no
//                  waiting) adds the partials and emits f32 and Q8_K output.
// Only float summation order differs from the sequential walk.
#include <algorithm>

#include "dc_common.cuh"
#include "dc_internal.h"
#include "dc_launch.cuh"

using namespace dc;

#define DC_TRY(expr)                       \
    do {                                   \
        int st_ = (expr);                  \
        if (st_ != DC_B200_OK) return st_; \
    } while (0)

#define ATT_MAX_GROUP 8  // query heads per kv head
#define ATT_TILE 32      // keys per score tile (two KV blocks)

struct AttnParams {
    const float* q;              // [T][n_head][128]
    const __half* k_arena;       // this layer
    const __half* v_arena;
    const int32_t* block_tables; // [max_seqs][max_blocks]
    int max_blocks;
    const int32_t* seq_ids;      // [T]
    const int32_t* positions;    // [T]
    int n_head, n_kv, T, nsplit;
    float scale;
    float* scores;               // [T][n_head][max_blocks*16]
    float* bmax;                 // [T][n_head][max_blocks]
    float* part_acc;             // [T][n_head][nsplit][128]
    float* part_d;               // [T][n_head][nsplit]
    int* tickets;                // [T][n_kv], zeroed once, self-resetting
    float* out;                  // optional [T][n_head][128]
    uint8_t* q8_out;             // optional Q8_K rows of out, blocks in fragment order
};

__device__ __forceinline__ void split_range(int pos, int split, int nsplit, int& n_blk, int& b0, int& b1) {
    n_blk = (pos + 1 + DC_KV_BLOCK - 1) / DC_KV_BLOCK;
    const int bps = (n_blk + nsplit - 1) / nsplit;
    b0 = min(n_blk, split * bps);
    b1 = min(n_blk, b0 + bps);
}

__global__ void __launch_bounds__(128) k_attn_scores(const AttnParams p) {
    // a q head as four 32-dim quarters 36 floats apart: the four lanes of a key read the same offset of
    // different quarters, which then fall into different banks
    __shared__ __align__(16) float sq[ATT_MAX_GROUP][4 * 36];
    __shared__ float sc[ATT_MAX_GROUP][ATT_TILE];
    __shared__ int s_blk[ATT_TILE / DC_KV_BLOCK];
    pdl_launch_dependents();
    const int split = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
    const int g = p.n_head / p.n_kv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // positions, sequence ids and block tables were settled before this step began, and K rows of earlier
    // positions are not written during it: the first tile's history rows are fetched while this kernel
    // still waits for the one that writes the new token's row and the q heads
    // (in an eager chain of steps the position may still be the previous step's here: everything is
    // recomputed after the wait and the early rows are dropped if the run moved)
    const int32_t* table = p.block_tables + (size_t)p.seq_ids[t] * p.max_blocks;
    uint4 kr0[4];
    bool pre = false;
    int pre_b0;
    {
        const int pos0 = p.positions[t];
        // rows written during this step: this token's, and those of earlier tokens of the same sequence
        // in a multi-token chunk; only rows before the first of them are safe to read early
        int stable = pos0;
        const int sid = p.seq_ids[t];
        for (int u = 0; u < p.T; ++u)
            if (p.seq_ids[u] == sid) stable = min(stable, p.positions[u]);
        int nb0, e1;
        split_range(pos0, split, p.nsplit, nb0, pre_b0, e1);
        const int key = warp * 8 + (lane >> 2), sub = lane & 3, blk = pre_b0 + key / DC_KV_BLOCK;
        const int kpos = pre_b0 * DC_KV_BLOCK + key;
        if (pos0 >= 0 && blk < e1 && kpos < stable) {
            const uint4* kp = reinterpret_cast<const uint4*>(
                p.k_arena + (((size_t)table[blk] * DC_KV_BLOCK + key % DC_KV_BLOCK) * p.n_kv + kvh) * 128 + sub * 32);
#pragma unroll
            for (int i = 0; i < 4; ++i) kr0[i] = kp[i];
            pre = true;
        }
    }
    pdl_wait();
    const int pos = *reinterpret_cast<const volatile int32_t*>(p.positions + t), ctx_len = pos + 1;
    int n_blk, b0, b1;
    split_range(pos, split, p.nsplit, n_blk, b0, b1);
    if (b0 != pre_b0) pre = false;
    if (b0 >= b1) return;
    for (int i = tid; i < g * 128; i += 128)
        sq[i >> 7][((i & 127) >> 5) * 36 + (i & 31)] = p.q[((size_t)t * p.n_head + kvh * g + (i >> 7)) * 128 + (i & 127)];
    __syncthreads();
    const size_t ctx_pad = (size_t)p.max_blocks * DC_KV_BLOCK;
    for (int blk = b0; blk < b1; blk += ATT_TILE / DC_KV_BLOCK) {
        if (tid < ATT_TILE / DC_KV_BLOCK) s_blk[tid] = (blk + tid < b1) ? table[blk + tid] : -1;
        __syncthreads();
        {   // 4 lanes per key, 32 dims per lane
            const int key = warp * 8 + (lane >> 2), sub = lane & 3;
            const int kpos = blk * DC_KV_BLOCK + key;
            const int pb = s_blk[key / DC_KV_BLOCK];
            const bool valid = pb >= 0 && kpos < ctx_len;
            float kf[32];
            if (valid) {
                const uint4* kp = reinterpret_cast<const uint4*>(
                    p.k_arena + (((size_t)pb * DC_KV_BLOCK + key % DC_KV_BLOCK) * p.n_kv + kvh) * 128 + sub * 32);
                const bool have = pre && blk == b0;   // fetched before the wait
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 u = have ? kr0[i] : kp[i];
                    const __half2* h2 = reinterpret_cast<const __half2*>(&u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __half22float2(h2[j]);
                        kf[i * 8 + 2 * j] = f.x;
                        kf[i * 8 + 2 * j + 1] = f.y;
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) kf[i] = 0.0f;
            }
            for (int h = 0; h < g; ++h) {
                float dot = 0.0f;
                const float4* qp = reinterpret_cast<const float4*>(&sq[h][sub * 36]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 qq = qp[i];
                    dot = fmaf(qq.x, kf[4 * i], dot);
                    dot = fmaf(qq.y, kf[4 * i + 1], dot);
                    dot = fmaf(qq.z, kf[4 * i + 2], dot);
                    dot = fmaf(qq.w, kf[4 * i + 3], dot);
                }
                dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                dot += __shfl_xor_sync(0xffffffffu, dot, 2);
                if (sub == 0) sc[h][key] = valid ? __fmul_rn(dot, p.scale) : -INFINITY;
            }
        }
        __syncthreads();
        // scores out (32 consecutive keys per head) and the two block maxima
        for (int i = tid; i < g * ATT_TILE; i += 128) {
            const int h = i / ATT_TILE, key = i % ATT_TILE;
            if (blk + key / DC_KV_BLOCK < b1)
                p.scores[((size_t)t * p.n_head + kvh * g + h) * ctx_pad + (size_t)blk * DC_KV_BLOCK + key] = sc[h][key];
        }
        if (tid < g * (ATT_TILE / DC_KV_BLOCK)) {
            const int h = tid / (ATT_TILE / DC_KV_BLOCK), bb = tid % (ATT_TILE / DC_KV_BLOCK);
            if (blk + bb < b1) {
                float mx = -1e30f;  // the reference's m_block starts at -1e30
#pragma unroll
                for (int k = 0; k < DC_KV_BLOCK; ++k) mx = fmaxf(mx, sc[h][bb * DC_KV_BLOCK + k]);
                p.bmax[((size_t)t * p.n_head + kvh * g + h) * p.max_blocks + blk + bb] = mx;
            }
        }
        __syncthreads();
    }
}

// Tail of both P.V kernels: the run's partials are in global memory; the last run of the (token, kv head)
// to get here sums all runs in run order, normalises and emits (no run waits for another).
__device__ __forceinline__ void attn_merge_tail(const AttnParams& p, int t, int kvh, int g, int tid, int warp, int lane,
                                                int& s_last) {
    // release: the CTA barrier puts every thread's partial before thread 0's ticket, whose release half publishes
    // them; acquire: the last run's thread 0 sees the other runs' partials through the ticket's acquire half, and
    // the CTA barrier passes that on
    __syncthreads();
    if (tid == 0) {
        int old;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p.tickets + t * p.n_kv + kvh), "r"(1) : "memory");
        const int last = old == p.nsplit - 1;
        if (last) p.tickets[t * p.n_kv + kvh] = 0;
        s_last = last;
    }
    __syncthreads();
    if (!s_last) return;
    // ---- last run of this (token, kv head): sum the runs in run order, normalise, emit.
    // One warp per 256 outputs (two heads) = one Q8_K block of the o-projection input.
    for (int pb2 = warp; pb2 < g / 2; pb2 += 4) {
        const int head = kvh * g + 2 * pb2 + (lane >> 4), d0 = (lane & 15) * 8;
        const size_t base = ((size_t)t * p.n_head + head) * p.nsplit;
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, den = 0.0f;
        for (int s0 = 0; s0 < p.nsplit; s0 += 8) {
            float dd[8];
            float4 a[8], c[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {   // eight runs' loads in flight, then added in run order
                const size_t bi = base + (s0 + j < p.nsplit ? s0 + j : 0);
                dd[j] = __ldcg(p.part_d + bi);
                a[j] = __ldcg(reinterpret_cast<const float4*>(p.part_acc + bi * 128 + d0));
                c[j] = __ldcg(reinterpret_cast<const float4*>(p.part_acc + bi * 128 + d0 + 4));
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (s0 + j < p.nsplit) {
                    den += dd[j];
                    v[0] += a[j].x; v[1] += a[j].y; v[2] += a[j].z; v[3] += a[j].w;
                    v[4] += c[j].x; v[5] += c[j].y; v[6] += c[j].z; v[7] += c[j].w;
                }
            }
        }
        const float inv = (den > 0.0f && isfinite(den)) ? __fdiv_rn(1.0f, __fadd_rn(den, 1e-6f)) : 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= inv;
        if (p.out) {
            float* o = p.out + ((size_t)t * p.n_head + head) * 128 + d0;
            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
        if (p.q8_out)
            quantize_block_q8f_regs(v, p.q8_out + ((size_t)t * (p.n_head / 2) + kvh * (g / 2) + pb2) * DC_Q8F_BYTES, lane);
    }
}

__global__ void __launch_bounds__(128) k_attn_pv(const AttnParams p) {
    __shared__ float s_p[ATT_MAX_GROUP][DC_KV_BLOCK];
    __shared__ float s_suffix[ATT_MAX_GROUP];
    __shared__ float s_m[ATT_MAX_GROUP], s_d[ATT_MAX_GROUP], s_alpha[ATT_MAX_GROUP];
    __shared__ int s_last;
    pdl_launch_dependents();
    pdl_wait();
    const int split = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
    const int g = p.n_head / p.n_kv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pos = p.positions[t], ctx_len = pos + 1;
    int n_blk, b0, b1;
    split_range(pos, split, p.nsplit, n_blk, b0, b1);
    const int32_t* table = p.block_tables + (size_t)p.seq_ids[t] * p.max_blocks;
    const size_t ctx_pad = (size_t)p.max_blocks * DC_KV_BLOCK;

    // ---- the reference's chain from all block maxima: m before this run, and the
    //      product of alpha_c over every block c >= b1 (blocks after this run)
    for (int h = warp; h < g; h += 4) {
        const float* bm = p.bmax + ((size_t)t * p.n_head + kvh * g + h) * p.max_blocks;
        float m_start = -1e30f;
        for (int b = lane; b < b0; b += 256) {   // eight loads in flight per lane
            float vb8[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) vb8[k] = b + 32 * k < b0 ? bm[b + 32 * k] : -1e30f;
#pragma unroll
            for (int k = 0; k < 8; ++k) m_start = fmaxf(m_start, vb8[k]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m_start = fmaxf(m_start, __shfl_xor_sync(0xffffffffu, m_start, o));
        float m_run = m_start;
        for (int b = b0 + lane; b < b1; b += 32) m_run = fmaxf(m_run, bm[b]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m_run = fmaxf(m_run, __shfl_xor_sync(0xffffffffu, m_run, o));
        // later blocks in chunks of 32: inclusive prefix max by shuffles, alpha per block, product
        float carry = m_run, suffix = 1.0f;
        for (int c0 = b1; c0 < n_blk; c0 += 32) {
            const int c = c0 + lane;
            float v = c < n_blk ? bm[c] : -1e30f;
            float incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl = fmaxf(incl, u);
            }
            float excl = __shfl_up_sync(0xffffffffu, incl, 1);
            if (lane == 0) excl = -1e30f;
            const float m_prev = fmaxf(carry, excl), m_new = fmaxf(carry, incl);
            float a = c < n_blk ? fast_exp_fma(m_prev - m_new) : 1.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a *= __shfl_xor_sync(0xffffffffu, a, o);
            suffix *= a;
            carry = fmaxf(carry, __shfl_sync(0xffffffffu, incl, 31));
        }
        if (lane == 0) {
            s_suffix[h] = suffix;
            s_m[h] = m_start;
            s_d[h] = 0.0f;
        }
    }
    float acc[ATT_MAX_GROUP];
#pragma unroll
    for (int h = 0; h < ATT_MAX_GROUP; ++h) acc[h] = 0.0f;
    __syncthreads();

    // ---- own blocks, one 16-key block at a time exactly as the reference walks them
    for (int blk = b0; blk < b1; ++blk) {
        const int pb = table[blk];
        const int nk = min(DC_KV_BLOCK, ctx_len - blk * DC_KV_BLOCK);
        {
            const int h = tid >> 4, key = tid & 15;  // 128 threads = 8 heads x 16 keys
            float s = -INFINITY;
            if (h < g && key < nk)
                s = p.scores[((size_t)t * p.n_head + kvh * g + h) * ctx_pad + (size_t)blk * DC_KV_BLOCK + key];
            float mx = fmaxf(s, -1e30f);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_prev = h < g ? s_m[h] : -1e30f;
            const float m_new = fmaxf(m_prev, mx);
            const float pr = (s == -INFINITY) ? 0.0f : fast_exp_fma(s - m_new);
            float ps = pr;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
            if (h < g) s_p[h][key] = pr;
            __syncwarp();
            if (h < g && key == 0) {
                const float alpha = fast_exp_fma(m_prev - m_new);
                s_alpha[h] = alpha;
                s_d[h] = s_d[h] * alpha + ps;
                s_m[h] = m_new;
            }
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < ATT_MAX_GROUP; ++h)
            if (h < g && s_alpha[h] != 1.0f) acc[h] *= s_alpha[h];
        const __half* vb = p.v_arena + ((size_t)pb * DC_KV_BLOCK * p.n_kv + kvh) * 128 + tid;
        // the block's 16 V values are requested together (rows beyond nk exist in the arena and are not used)
        __half vv[DC_KV_BLOCK];
#pragma unroll
        for (int key = 0; key < DC_KV_BLOCK; ++key) vv[key] = vb[(size_t)key * p.n_kv * 128];
#pragma unroll
        for (int key = 0; key < DC_KV_BLOCK; ++key) {
            if (key < nk) {
                const float v = __half2float(vv[key]);
#pragma unroll
                for (int h = 0; h < ATT_MAX_GROUP; ++h)
                    if (h < g) acc[h] = fmaf(s_p[h][key], v, acc[h]);
            }
        }
        __syncthreads();
    }
    // ---- partials scaled by the alphas of all later blocks
#pragma unroll
    for (int h = 0; h < ATT_MAX_GROUP; ++h) {
        if (h < g) {
            const size_t idx = ((size_t)t * p.n_head + kvh * g + h) * p.nsplit + split;
            p.part_acc[idx * 128 + tid] = acc[h] * s_suffix[h];
            if (tid == 0) p.part_d[idx] = s_d[h] * s_suffix[h];
        }
    }
    attn_merge_tail(p, t, kvh, g, tid, warp, lane, s_last);
}

// Same result as k_attn_pv for runs of at most ATT_MAX_RUN KV blocks, organised for latency: every
// block's running maximum and rescale factor follow from the block maxima alone, so they are computed
// for the whole run first (one batched load, prefix maxima by shuffles); then all exponentials of the
// run at once; then one pass over the keys with no CTA barrier inside.
#define ATT_MAX_RUN 64
__global__ void __launch_bounds__(128) k_attn_pv_run(const AttnParams p) {
    __shared__ __align__(16) float s_pw[ATT_MAX_GROUP * ATT_MAX_RUN * DC_KV_BLOCK];   // scores of the run, then exponentials
    __shared__ float s_mnew[ATT_MAX_GROUP][ATT_MAX_RUN], s_alpha[ATT_MAX_GROUP][ATT_MAX_RUN], s_ps[ATT_MAX_GROUP][ATT_MAX_RUN];
    __shared__ float s_suffix[ATT_MAX_GROUP];
    __shared__ int s_blk[ATT_MAX_RUN];
    __shared__ int s_last;
    pdl_launch_dependents();
    pdl_wait();
    const int split = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
    const int g = p.n_head / p.n_kv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pos = p.positions[t], ctx_len = pos + 1;
    int n_blk, b0, b1;
    split_range(pos, split, p.nsplit, n_blk, b0, b1);
    const int32_t* table = p.block_tables + (size_t)p.seq_ids[t] * p.max_blocks;
    const size_t ctx_pad = (size_t)p.max_blocks * DC_KV_BLOCK;
    const int nb = b1 - b0, stride = nb * DC_KV_BLOCK;
    for (int i = tid; i < g * stride; i += 128) {
        const int h = i / stride, k = i - h * stride;
        s_pw[i] = p.scores[((size_t)t * p.n_head + kvh * g + h) * ctx_pad + (size_t)b0 * DC_KV_BLOCK + k];
    }
    for (int i = tid; i < nb; i += 128) s_blk[i] = table[b0 + i];
    for (int h = warp; h < g; h += 4) {
        const float* bm = p.bmax + ((size_t)t * p.n_head + kvh * g + h) * p.max_blocks;
        float carry = -1e30f, suffix = 1.0f;
        for (int s0 = 0; s0 < n_blk; s0 += 256) {
            float vb[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = s0 + 32 * k + lane;
                vb[k] = c < n_blk ? bm[c] : -1e30f;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c0 = s0 + 32 * k, c = c0 + lane;
                if (c0 >= n_blk) break;
                if (c0 + 32 <= b0) {   // wholly before the run: only the running maximum
                    float mx = vb[k];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    carry = fmaxf(carry, mx);
                    continue;
                }
                float incl = vb[k];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl = fmaxf(incl, u);
                }
                float excl = __shfl_up_sync(0xffffffffu, incl, 1);
                if (lane == 0) excl = -1e30f;
                const float m_prev = fmaxf(carry, excl), m_new = fmaxf(carry, incl);
                const float a = (c >= b0 && c < n_blk) ? fast_exp_fma(m_prev - m_new) : 1.0f;
                if (c >= b0 && c < b1) {
                    s_mnew[h][c - b0] = m_new;
                    s_alpha[h][c - b0] = a;
                }
                if (c0 + 32 > b1) {   // the chunk reaches past the run: those factors go into the suffix
                    float later = c >= b1 ? a : 1.0f;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) later *= __shfl_xor_sync(0xffffffffu, later, o);
                    suffix *= later;
                }
                carry = fmaxf(carry, __shfl_sync(0xffffffffu, incl, 31));
            }
        }
        if (lane == 0) s_suffix[h] = suffix;
    }
    __syncthreads();
    // exponentials: 16 lanes per (head, block)
    for (int base = 0; base < g * nb; base += 8) {
        const int pair = base + (tid >> 4), key = tid & 15;
        const bool in = pair < g * nb;
        const int h = in ? pair / nb : 0, bl = in ? pair - h * nb : 0;
        const int nk = min(DC_KV_BLOCK, ctx_len - (b0 + bl) * DC_KV_BLOCK);
        const float s = (in && key < nk) ? s_pw[h * stride + bl * DC_KV_BLOCK + key] : -INFINITY;
        const float pr = (s == -INFINITY) ? 0.0f : fast_exp_fma(s - s_mnew[h][bl]);
        float ps = pr;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
        if (in) {
            s_pw[h * stride + bl * DC_KV_BLOCK + key] = pr;
            if (key == 0) s_ps[h][bl] = ps;
        }
    }
    __syncthreads();
    // thread = dim; one accumulator per head; thread h also carries head h's denominator
    float acc[ATT_MAX_GROUP];
#pragma unroll
    for (int h = 0; h < ATT_MAX_GROUP; ++h) acc[h] = 0.0f;
    float den = 0.0f;
    // a block's 16 V values are requested together, one block ahead of the FMAs (rows beyond nk exist in
    // the arena and are not used)
    __half vn[DC_KV_BLOCK];
    if (nb > 0) {
        const __half* vb = p.v_arena + ((size_t)s_blk[0] * DC_KV_BLOCK * p.n_kv + kvh) * 128 + tid;
#pragma unroll
        for (int key = 0; key < DC_KV_BLOCK; ++key) vn[key] = vb[(size_t)key * p.n_kv * 128];
    }
    for (int bl = 0; bl < nb; ++bl) {
        const int nk = min(DC_KV_BLOCK, ctx_len - (b0 + bl) * DC_KV_BLOCK);
        __half vv[DC_KV_BLOCK];
#pragma unroll
        for (int key = 0; key < DC_KV_BLOCK; ++key) vv[key] = vn[key];
        if (bl + 1 < nb) {
            const __half* vb = p.v_arena + ((size_t)s_blk[bl + 1] * DC_KV_BLOCK * p.n_kv + kvh) * 128 + tid;
#pragma unroll
            for (int key = 0; key < DC_KV_BLOCK; ++key) vn[key] = vb[(size_t)key * p.n_kv * 128];
        }
        if (tid < g) den = den * s_alpha[tid][bl] + s_ps[tid][bl];
#pragma unroll
        for (int h = 0; h < ATT_MAX_GROUP; ++h)
            if (h < g && s_alpha[h][bl] != 1.0f) acc[h] *= s_alpha[h][bl];
        float vf[DC_KV_BLOCK];
#pragma unroll
        for (int key = 0; key < DC_KV_BLOCK; ++key) vf[key] = __half2float(vv[key]);
        // per head: the block's 16 exponentials in four 128-bit loads, then the FMA chain in key order
#pragma unroll
        for (int h = 0; h < ATT_MAX_GROUP; ++h) {
            if (h < g) {
                float pp[DC_KV_BLOCK];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<float4*>(&pp[4 * q]) =
                        *reinterpret_cast<const float4*>(&s_pw[h * stride + bl * DC_KV_BLOCK + 4 * q]);
#pragma unroll
                for (int key = 0; key < DC_KV_BLOCK; ++key)
                    if (key < nk) acc[h] = fmaf(pp[key], vf[key], acc[h]);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < ATT_MAX_GROUP; ++h) {
        if (h < g) {
            const size_t idx = ((size_t)t * p.n_head + kvh * g + h) * p.nsplit + split;
            p.part_acc[idx * 128 + tid] = acc[h] * s_suffix[h];
        }
    }
    if (tid < g) p.part_d[((size_t)t * p.n_head + kvh * g + tid) * p.nsplit + split] = den * s_suffix[tid];
    attn_merge_tail(p, t, kvh, g, tid, warp, lane, s_last);
}

// ------------------------------------------------------- one kernel, a cluster per (token, kv head)
// What bounds decode attention at these lengths is not its bytes (4.7 MB of K and V at 2304 keys: 0.7 us of HBM) but the chain of
// global round trips between score, P.V and merge kernels.  Here the CTAs of a cluster share a sequence's runs and exchange
// block maxima and partial sums through each other's shared memory: K and V rows of earlier positions are copied to shared memory while
// this kernel still waits for its predecessor, scores never leave the SM, and the merge reads all partials at once.
// The runs, and the order of every float operation, are those of k_attn_scores and k_attn_pv_run, so the results are theirs bit for bit
// and which kernels serve a call is a matter of speed alone: a key's product is four chains of 32 dimensions, a run walks its keys in
// order and multiplies the reference's alpha onto its accumulator at every block, the alphas of later blocks are multiplied 32 at a
// time, and the merge adds the runs in order.  (Q8_K rounding downstream turns a difference in the last bit into one of 1 % in the logits
// of a random model, so that another order of sums would not be told from an error.)
// With `fuse.qkv` the kernel also norms and rotates the q heads (every CTA its own copy) and writes the new token's K and V rows
// (k_qknorm_rope_kv); the tokens of such a step belong to different sequences.
// What bounds it: the launch's dependency gap, then the latency of its phases (scores 3 to 4 thousand cycles of 16 at one token and 2000
// keys, P.V as long), in which instructions met for the first time cost as much as the arithmetic: loops over heads, blocks and runs
// stay rolled.  32 Q / 4 KV heads, 2000 keys, one token, a step of three layers: 178 us; with the split kernels and k_qknorm_rope_kv 260;
// 171 with keys dealt out over the threads in an order of sums that is not the split kernels'.
#define AC_THREADS 256
#define AC_CAP 48              // KV blocks a CTA holds at most
#define AC_SMEM (220 * 1024)
#define AC_Q_PITCH 144         // floats of a q head: four quarters 36 apart, which fall into different banks

// The runs of a sequence (split_range's, the empty ones left out) that CTA `rank` of C works on, and its blocks.
struct AcRuns {
    int n_blk, bps, n_run, rpc;      // blocks, blocks of a run, runs, runs of a CTA
    int r0, r1, b0, b1;
    __device__ __forceinline__ void set(int pos, int rank, int C, int nsplit) {
        n_blk = (pos + 1 + DC_KV_BLOCK - 1) / DC_KV_BLOCK;
        bps = max(1, (n_blk + nsplit - 1) / nsplit);
        n_run = (n_blk + bps - 1) / bps;
        rpc = max(1, (n_run + C - 1) / C);
        r0 = min(n_run, rank * rpc);
        r1 = min(n_run, r0 + rpc);
        b0 = min(n_blk, r0 * bps);
        b1 = min(n_blk, r1 * bps);
    }
};

__device__ __forceinline__ uint32_t ac_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ac_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of `mine` in CTA `rank`'s shared memory, and a load from such an address
__device__ __forceinline__ uint32_t ac_map(const float* mine, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(mine)), "r"(rank));
    return a;
}
__device__ __forceinline__ float ac_load(uint32_t a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
// place of 16-byte piece i of a key's K row: piece 4 q + i of quarter q at 4 i + q, so that eight lanes (four quarters of two
// neighbouring keys) fall on distinct banks
__device__ __forceinline__ int ac_piece(int key, int i) { return key * 256 + ((((i & 3) << 2 | i >> 2) ^ ((key & 1) << 2)) << 4); }
__device__ __forceinline__ void ac_copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One head of 128 values by one warp: RMSNorm (w4 given) and rotation of interleaved pairs (c given), as k_qknorm_rope_kv.
__device__ __forceinline__ float4 ac_norm_rope(const float* src, bool norm, float4 w4, bool turn, float4 c, float eps, int lane) {
    const float4 v4 = __ldcg(reinterpret_cast<const float4*>(src) + lane);
    float v[4] = {v4.x, v4.y, v4.z, v4.w};
    if (norm) {
        double ss = (double)v[0] * v[0] + (double)v[1] * v[1] + (double)v[2] * v[2] + (double)v[3] * v[3];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float mean = (float)(ss / 128.0);
        const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
        v[0] = __fmul_rn(__fmul_rn(v[0], scale), w4.x);
        v[1] = __fmul_rn(__fmul_rn(v[1], scale), w4.y);
        v[2] = __fmul_rn(__fmul_rn(v[2], scale), w4.z);
        v[3] = __fmul_rn(__fmul_rn(v[3], scale), w4.w);
    }
    if (turn) {
        const float a0 = __fsub_rn(__fmul_rn(v[0], c.x), __fmul_rn(v[1], c.y)), a1 = __fadd_rn(__fmul_rn(v[0], c.y), __fmul_rn(v[1], c.x));
        const float b0 = __fsub_rn(__fmul_rn(v[2], c.z), __fmul_rn(v[3], c.w)), b1 = __fadd_rn(__fmul_rn(v[2], c.w), __fmul_rn(v[3], c.z));
        v[0] = a0; v[1] = a1; v[2] = b0; v[3] = b1;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ uint2 ac_half4(float4 v) {
    const __half2 lo = __halves2half2(__float2half_rn(v.x), __float2half_rn(v.y)), hi = __halves2half2(__float2half_rn(v.z), __float2half_rn(v.w));
    uint2 r;
    r.x = *reinterpret_cast<const uint32_t*>(&lo);
    r.y = *reinterpret_cast<const uint32_t*>(&hi);
    return r;
}

// P.V of one run (the j-th of this CTA's): H heads from h0 on, D dimensions from d0 on a thread; the results times the alphas of all later
// blocks.
template <int H, int D>
__device__ __forceinline__ void ac_pv(const AcRuns& R, const uint8_t* sKV, const float* sP, const float* sAl, const float* sSuf, int j, int h0, int d0, int g,
                                      int cap, int ps, int keys, float (&a)[H][D]) {
    constexpr int N = H * D > 4 ? 4 : 16;      // keys whose loads are in flight together
    const int end = min(R.b1 - R.b0, (j + 1) * R.bps);
    auto row = [&](const uint8_t* v, float (&f)[D]) {
        if constexpr (D == 4) {
            const uint2 u = *reinterpret_cast<const uint2*>(v);
            const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), y = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
            f[0] = x.x, f[1] = x.y, f[2] = y.x, f[3] = y.y;
        } else {
            const float2 x = __half22float2(*reinterpret_cast<const __half2*>(v));
            f[0] = x.x, f[1] = x.y;
        }
    };
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int d = 0; d < D; ++d) a[h][d] = 0.0f;
#pragma unroll 1
    for (int bl = j * R.bps; bl < end; ++bl) {
        const uint8_t* v = sKV + bl * DC_KV_BLOCK * 256 + d0 * 2;
        const float* pp = sP + h0 * ps + bl * DC_KV_BLOCK;
        const int nk = keys - bl * DC_KV_BLOCK;      // (16 or more, but for the sequence's last block)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const float al = sAl[(h0 + h) * cap + bl];
#pragma unroll
            for (int d = 0; d < D; ++d) a[h][d] = __fmul_rn(a[h][d], al);
        }
        if (nk >= DC_KV_BLOCK) {
#pragma unroll 1
            for (int q = 0; q < DC_KV_BLOCK; q += N) {
                float4 x[H][N / 4];
                float f[N][D];
#pragma unroll
                for (int k = 0; k < N; ++k) row(v + (q + k) * 256, f[k]);
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int k = 0; k < N / 4; ++k) x[h][k] = *reinterpret_cast<const float4*>(pp + h * ps + q + 4 * k);
#pragma unroll
                for (int k = 0; k < N; ++k)
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float4& y = x[h][k / 4];
                        const float w = k % 4 == 0 ? y.x : k % 4 == 1 ? y.y : k % 4 == 2 ? y.z : y.w;
#pragma unroll
                        for (int d = 0; d < D; ++d) a[h][d] = fmaf(w, f[k][d], a[h][d]);
                    }
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < nk; ++k) {
                float f[D];
                row(v + k * 256, f);
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const float w = pp[h * ps + k];
#pragma unroll
                    for (int d = 0; d < D; ++d) a[h][d] = fmaf(w, f[d], a[h][d]);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const float f = sSuf[j * g + h0 + h];
#pragma unroll
        for (int d = 0; d < D; ++d) a[h][d] = __fmul_rn(a[h][d], f);
    }
}
// All of this CTA's runs by the CTA's four groups of threads.  Several runs: a group takes a run, its warps half of the heads each, and
// leaves the sums where the run's V rows were, which nobody else reads.  At most one run: the groups share its heads, and the
// sums go to `one`.
template <int G>
__device__ __forceinline__ void ac_pv_all(const AcRuns& R, uint8_t* sKV, const float* sP, const float* sAl, const float* sSuf, float* one, int cap, int rcap,
                                          int ps, int keys) {
    const int kg = threadIdx.x >> 6, nr = R.r1 - R.r0;
    if (rcap == 1) {
        constexpr int H = G == 8 || G == 6 ? 2 : 1;
        const int d0 = 2 * (threadIdx.x & 63);
        if (nr > 0 && kg < G / H) {
            float a[H][2];
            ac_pv<H, 2>(R, sKV, sP, sAl, sSuf, 0, kg * H, d0, G, cap, ps, keys, a);
#pragma unroll
            for (int h = 0; h < H; ++h) *reinterpret_cast<float2*>(one + (kg * H + h) * 128 + d0) = make_float2(a[h][0], a[h][1]);
        }
        return;
    }
    constexpr int H = G / 2;
    const int h0 = (threadIdx.x >> 5 & 1) * H, d0 = 4 * (threadIdx.x & 31);
    for (int j = kg; j < nr; j += AC_THREADS / 64) {
        float a[H][4];
        ac_pv<H, 4>(R, sKV, sP, sAl, sSuf, j, h0, d0, G, cap, ps, keys, a);
        asm volatile("bar.sync %0, 64;" ::"r"(1 + kg) : "memory");      // the group has read the run's V rows
        float* to = reinterpret_cast<float*>(sKV + (size_t)j * R.bps * DC_KV_BLOCK * 256) + h0 * 128 + d0;
#pragma unroll
        for (int h = 0; h < H; ++h) *reinterpret_cast<float4*>(to + h * 128) = make_float4(a[h][0], a[h][1], a[h][2], a[h][3]);
    }
}

// C: CTAs of a cluster.  cap, rcap: KV blocks and runs that a CTA holds at most.  hs: clusters that share a kv head's query heads.
template <int C>
__global__ void __launch_bounds__(AC_THREADS, 2) k_attn_cluster(const AttnParams p, const dc_attn_fuse fuse, const int cap, const int rcap, const int hs) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int32_t sTab[AC_CAP];                               // ids of this CTA's KV blocks
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)ac_rank(), kvh = blockIdx.x / (C * hs), part = blockIdx.x / C % hs, t = blockIdx.y, g = p.n_head / p.n_kv / hs;
    const int head0 = (kvh * hs + part) * g;                       // first of this cluster's query heads
    const int ps = cap * DC_KV_BLOCK + 4;                          // floats between heads' scores: eight heads' pieces on distinct banks
    uint8_t* sKV = smem;                                           // K rows, after the scores V rows: [key][256]
    float* sP = reinterpret_cast<float*>(sKV + cap * DC_KV_BLOCK * 256);   // [head][ps] scores, then exponentials
    float* sQ = sP + g * ps;                                       // [head][AC_Q_PITCH]
    float* sDen = sQ + g * AC_Q_PITCH;                             // [run][head], read by the other CTAs, as is the next
    float* sBm = sDen + rcap * g;                                  // [head][block] block maximum
    float* sM = sBm + g * cap;                                     // [head][block] the maximum to take exponents against, then the exponentials' sum
    float* sAl = sM + g * cap;                                     // [head][block] alpha
    float* sSuf = sAl + g * cap;                                   // [run][head] product of the alphas of all later blocks
    pdl_launch_dependents();
    const int sid = p.seq_ids[t];
    const int32_t* table = p.block_tables + (size_t)sid * p.max_blocks;
    const size_t row = (size_t)p.n_kv * 128;                       // elements per token
    const uint32_t aKV = smem_u32(sKV);
    // K rows of keys [from, to), of which this CTA's first is k0
    auto load_k = [&](int k0, int from, int to) {
        for (int key = from + (tid >> 4); key < to; key += AC_THREADS / 16) {
            const size_t off = ((size_t)table[key / DC_KV_BLOCK] * DC_KV_BLOCK + key % DC_KV_BLOCK) * row + kvh * 128 + (tid & 15) * 8;
            ac_copy16(aKV + ac_piece(key - k0, tid & 15), p.k_arena + off);
        }
    };
    // positions, sequence ids and block tables were settled before this step began, and rows of earlier positions are not written
    // during it (in an eager chain of steps the position may still be the previous step's here: everything is looked at again after
    // the wait)
    const int pos0 = p.positions[t];
    int stable = pos0;
    if (!fuse.qkv)
        for (int u = 0; u < p.T; ++u)
            if (p.seq_ids[u] == sid) stable = min(stable, p.positions[u]);
    AcRuns R;
    R.set(pos0, rank, C, p.nsplit);
    const bool early = pos0 >= 0 && R.b1 - R.b0 <= cap;
    if (early) {
        const int from = R.b0 * DC_KV_BLOCK, to = min(R.b1 * DC_KV_BLOCK, stable);
        load_k(from, from, to);
        // V's turn in the shared buffer comes after the scores; until then its rows, two lines each, come from HBM into L2
        // (a 48-layer step at 2050 keys: 0.8 % of it)
        for (int i = tid; i < 2 * (to - from); i += AC_THREADS) {
            const int key = from + (i >> 1);
            const __half* v = p.v_arena + ((size_t)table[key / DC_KV_BLOCK] * DC_KV_BLOCK + key % DC_KV_BLOCK) * row + kvh * 128 + (i & 1) * 64;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(v));
        }
    }
    auto turn_at = [&](int at) {
        const int rp = at < 0 ? 0 : (fuse.max_pos > 0 && at >= fuse.max_pos) ? fuse.max_pos - 1 : at;
        return reinterpret_cast<const float4*>(fuse.cos_sin + (size_t)rp * 128)[lane];
    };
    float4 qw = make_float4(0.f, 0.f, 0.f, 0.f), kw = qw, turn = qw;
    if (fuse.qkv) {
        if (fuse.qn_w) qw = reinterpret_cast<const float4*>(fuse.qn_w)[lane];
        if (fuse.kn_w) kw = reinterpret_cast<const float4*>(fuse.kn_w)[lane];
        turn = turn_at(pos0);
    }
    pdl_wait();
    const int pos = *reinterpret_cast<const volatile int32_t*>(p.positions + t);
    if (pos != pos0) R.set(pos, rank, C, p.nsplit);
    const int k0 = R.b0 * DC_KV_BLOCK, nbl = R.b1 - R.b0, nr = R.r1 - R.r0, keys = max(0, min(pos + 1, R.b1 * DC_KV_BLOCK) - k0);
    {
        const bool same = early && pos == pos0;
        if (tid < nbl) sTab[tid] = table[R.b0 + tid];
        if (!same) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        load_k(k0, same ? max(k0, stable) : k0, k0 + keys - (fuse.qkv && k0 + keys == pos + 1 ? 1 : 0));
    }
    uint2 new_v = make_uint2(0u, 0u);     // the new token's V row (warp 7), which has to wait for the K rows to go
    const bool mine = fuse.qkv && keys > 0 && k0 + keys == pos + 1;
    // a lane's four values of a q head: dimensions 4 lane .. 4 lane + 3
    auto q_at = [&](int h, int l) { return reinterpret_cast<float4*>(sQ + h * AC_Q_PITCH + (l >> 3) * 36) + (l & 7); };
    if (fuse.qkv) {
        const float* src = fuse.qkv + (size_t)t * (p.n_head + 2 * p.n_kv) * 128;
        if (pos != pos0) turn = turn_at(pos);
        if (warp < g) *q_at(warp, lane) = ac_norm_rope(src + (head0 + warp) * 128, fuse.qn_w != nullptr, qw, true, turn, fuse.eps, lane);
        if (mine && warp >= 6) {       // the new token's rows: to the cache and to this CTA's tiles
            const bool is_k = warp == 6;
            const float4 v = ac_norm_rope(src + (p.n_head + (is_k ? 0 : p.n_kv) + kvh) * 128, is_k && fuse.kn_w, kw, is_k, turn, fuse.eps, lane);
            const uint2 hv = ac_half4(v);
            const size_t off = ((size_t)table[pos / DC_KV_BLOCK] * DC_KV_BLOCK + pos % DC_KV_BLOCK) * row + kvh * 128 + 4 * lane;
            if (part == 0) *reinterpret_cast<uint2*>(const_cast<__half*>(is_k ? p.k_arena : p.v_arena) + off) = hv;
            if (is_k) *reinterpret_cast<uint2*>(sKV + ac_piece(pos - k0, lane >> 1) + 8 * (lane & 1)) = hv;
            else new_v = hv;
        }
    } else {
        for (int i = tid; i < g * 32; i += AC_THREADS) *q_at(i >> 5, i & 31) = reinterpret_cast<const float4*>(p.q + ((size_t)t * p.n_head + head0) * 128)[i];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- scores: a warp keeps two heads' queries in registers, a quarter a lane, and takes eight keys at a time, four lanes each (queries
    // read again for every key had the shared memory's bandwidth as their bound)
    if (const int pairs = g / 2, turns = 8 / pairs; warp < pairs * turns) {
        const int h0 = 2 * (warp % pairs), sub = lane & 3;
        float q[2][32];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 x = reinterpret_cast<const float4*>(sQ + (h0 + h) * AC_Q_PITCH + sub * 36)[i];
                q[h][4 * i] = x.x, q[h][4 * i + 1] = x.y, q[h][4 * i + 2] = x.z, q[h][4 * i + 3] = x.w;
            }
#pragma unroll 1
        for (int key = warp / pairs * 8 + (lane >> 2); key < nbl * DC_KV_BLOCK; key += 8 * turns) {      // (16 keys a block: whole warps)
            float d[2] = {0.0f, 0.0f};
            uint4 u[4];      // (the rows after the last key's are read as whatever they hold and not used)
#pragma unroll
            for (int i = 0; i < 4; ++i) u[i] = *reinterpret_cast<const uint4*>(sKV + ac_piece(key, 4 * sub + i));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __half2* h2 = reinterpret_cast<const __half2*>(&u[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __half22float2(h2[j]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) d[h] = fmaf(q[h][8 * i + 2 * j], f.x, d[h]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) d[h] = fmaf(q[h][8 * i + 2 * j + 1], f.y, d[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                d[h] += __shfl_xor_sync(0xffffffffu, d[h], 1);
                d[h] += __shfl_xor_sync(0xffffffffu, d[h], 2);
            }
            if (sub < 2) sP[(h0 + sub) * ps + key] = key < keys ? __fmul_rn(sub ? d[1] : d[0], p.scale) : -INFINITY;
        }
    }
    __syncthreads();
    // the V rows follow into the same memory while the block maxima make their way
    for (int key = tid >> 4; key < keys - (mine ? 1 : 0); key += AC_THREADS / 16) {
        const size_t off = ((size_t)sTab[key / DC_KV_BLOCK] * DC_KV_BLOCK + key % DC_KV_BLOCK) * row + kvh * 128 + (tid & 15) * 8;
        ac_copy16(aKV + key * 256 + (tid & 15) * 16, p.v_arena + off);
    }
    if (mine && warp == 7) *reinterpret_cast<uint2*>(sKV + (pos - k0) * 256 + 8 * lane) = new_v;
    // sixteen lanes per (head, block), neighbouring groups on neighbouring heads
    const int lg = g > 4 ? 3 : g > 2 ? 2 : 1, hx = (tid >> 4) & ((1 << lg) - 1), bx = tid >> 4 >> lg, nbx = (nbl + (16 >> lg) - 1) >> (4 - lg) << (4 - lg);
    for (int bl = bx; bl < nbx; bl += 16 >> lg) {
        const bool in = hx < g && bl < nbl;
        float mx = in ? fmaxf(sP[hx * ps + bl * DC_KV_BLOCK + (tid & 15)], -1e30f) : -1e30f;  // the reference's m_block starts at -1e30
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (in && (tid & 15) == 0) sBm[hx * cap + bl] = mx;
    }
    ac_sync();
    // ---- the chain of a head by a warp, a lane per block, 32 blocks of the sequence at a time (as k_attn_pv_run)
    if (warp < g && nr > 0) {
        const int per = R.rpc * R.bps;         // blocks of a CTA
        const float inv = __frcp_rn((float)per);
        float carry = -1e30f, suf = 1.0f;      // lane j: the product of the j-th run
        auto block_max = [&](int c) {
            const int owner = (int)(((float)c + 0.5f) * inv);      // c / per
            return c < R.n_blk ? ac_load(ac_map(sBm + warp * cap + (c - owner * per), owner)) : -1e30f;
        };
        float next = block_max(lane);
#pragma unroll 1
        for (int c0 = 0; c0 < R.n_blk; c0 += 32) {
            const int c = c0 + lane;
            float incl = next;
            next = block_max(c + 32);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl = fmaxf(incl, u);
            }
            float excl = __shfl_up_sync(0xffffffffu, incl, 1);
            if (lane == 0) excl = -1e30f;
            const float m_prev = fmaxf(carry, excl), m_new = fmaxf(carry, incl);
            carry = fmaxf(carry, __shfl_sync(0xffffffffu, incl, 31));
            const float a = (c >= R.b0 && c < R.n_blk) ? fast_exp_fma(m_prev - m_new) : 1.0f;
            if (c >= R.b0 && c < R.b1) {
                sM[warp * cap + c - R.b0] = m_new;
                sAl[warp * cap + c - R.b0] = a;
            }
            if (__all_sync(0xffffffffu, a == 1.0f)) continue;      // factors of one leave a product as it is
#pragma unroll 1
            for (int j = 0; j < nr; ++j) {
                const int after = (R.r0 + j + 1) * R.bps;
                if (c0 + 32 <= after) break;
                float later = c >= after ? a : 1.0f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) later *= __shfl_xor_sync(0xffffffffu, later, o);
                if (lane == j) suf *= later;
            }
        }
        if (lane < nr) sSuf[lane * g + warp] = suf;
    }
    __syncthreads();
    // ---- exponentials and their sums over a block
#pragma unroll 2
    for (int bl = bx; bl < nbx; bl += 16 >> lg) {
        const bool in = hx < g && bl < nbl;
        float* at = sP + hx * ps + bl * DC_KV_BLOCK + (tid & 15);
        const float s = in ? *at : -INFINITY;
        const float pr = s == -INFINITY ? 0.0f : fast_exp_fma(s - sM[hx * cap + bl]);
        float sum = pr;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (in) {
            *at = pr;
            if ((tid & 15) == 0) sM[hx * cap + bl] = sum;      // (its sixteen readers are done with the maximum)
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- denominators of the runs by the last group of threads, which P.V keeps least busy (nr * g <= 64)
    if (tid >= AC_THREADS - 64 && tid - (AC_THREADS - 64) < nr * g) {
        const int i = tid - (AC_THREADS - 64), j = i / g, h = i - j * g, end = min(nbl, (j + 1) * R.bps);
        float den = 0.0f;
        for (int bl = j * R.bps; bl < end; ++bl) den = fmaf(den, sAl[h * cap + bl], sM[h * cap + bl]);
        sDen[i] = __fmul_rn(den, sSuf[i]);
    }
    if (g == 8) ac_pv_all<8>(R, sKV, sP, sAl, sSuf, sQ, cap, rcap, ps, keys);
    else if (g == 6) ac_pv_all<6>(R, sKV, sP, sAl, sSuf, sQ, cap, rcap, ps, keys);
    else if (g == 4) ac_pv_all<4>(R, sKV, sP, sAl, sSuf, sQ, cap, rcap, ps, keys);
    else ac_pv_all<2>(R, sKV, sP, sAl, sSuf, sQ, cap, rcap, ps, keys);
    ac_sync();
    // ---- merge: CTA r writes the head pair r, the 256 values of one Q8_K block of the o-projection's input, a thread a value, the runs
    // added in order
    float* sOut = rcap == 1 ? reinterpret_cast<float*>(sKV) : sQ;      // (whichever does not hold the sums)
    if (rank < g / 2) {
        const int head = 2 * rank + (tid >> 7), d = tid & 127;
        const float* sums = rcap == 1 ? sQ : reinterpret_cast<const float*>(sKV);
        const int step = R.bps * DC_KV_BLOCK * 64;      // floats between two runs' sums
        const float per = __frcp_rn((float)R.rpc);
        float acc = 0.0f, den = 0.0f;
#pragma unroll 1
        for (int r0 = 0; r0 < R.n_run; r0 += 8) {
            float x[8], y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {      // eight runs' loads in flight
                const int r = min(r0 + i, R.n_run - 1), owner = (int)(((float)r + 0.5f) * per), j = r - owner * R.rpc;
                const uint32_t base = ac_map(sums, owner);
                x[i] = ac_load(base + (uint32_t)(j * step + head * 128 + d) * 4u);
                y[i] = ac_load(base + (uint32_t)(sDen - sums + j * g + head) * 4u);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (r0 + i < R.n_run) {
                    acc += x[i];
                    den += y[i];
                }
        }
        const float inv = (den > 0.0f && isfinite(den)) ? __fdiv_rn(1.0f, __fadd_rn(den, 1e-6f)) : 0.0f;
        acc *= inv;
        if (p.out) p.out[((size_t)t * p.n_head + head0 + head) * 128 + d] = acc;
        sOut[tid] = acc;
    }
    ac_sync();      // nobody leaves while its shared memory is read (and sOut is whole)
    if (p.q8_out && rank < g / 2 && warp == 0) {
        const float4 x = reinterpret_cast<const float4*>(sOut)[2 * lane], y = reinterpret_cast<const float4*>(sOut)[2 * lane + 1];
        const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        quantize_block_q8f_regs(v, p.q8_out + ((size_t)t * (p.n_head / 2) + head0 / 2 + rank) * DC_Q8F_BYTES, lane);
    }
}

// Blocks and runs that a CTA of a cluster of C meets at most, for any length up to max_blocks: with runs of a given length the longest
// sequence has the most runs, and all lengths but the longest come with all nsplit runs.
struct AcPlan {
    int cap, rcap;
    AcPlan(int C, int max_blocks, int nsplit) {
        auto up = [](int a, int b) { return (a + b - 1) / b; };
        const int bps = up(max_blocks, nsplit);
        cap = up(up(max_blocks, bps), C) * bps;
        if (bps > 1) cap = std::max(cap, up(nsplit, C) * (bps - 1));
        rcap = up(std::min(nsplit, max_blocks), C);
    }
    size_t smem(int g) const {
        return (size_t)cap * DC_KV_BLOCK * 256 + (size_t)g * (cap * DC_KV_BLOCK + 4 + AC_Q_PITCH + 2 * rcap + 3 * cap) * 4;
    }
};
// few tokens: two clusters share a kv head's query heads, as long as there is an SM for every CTA
static int attn_head_split(int C, int T, int n_kv, int g) { return g % 4 == 0 && 2 * T * n_kv * C <= 128 ? 2 : 1; }
static bool attn_cluster_fits(int C, int T, int n_kv, int g, int max_blocks, int nsplit) {
    const AcPlan plan(C, max_blocks, nsplit);
    // a thread for each of 8 x 8 denominators; runs longer than ATT_MAX_RUN take k_attn_pv, which multiplies alphas in another order
    if (plan.rcap > 8 || (max_blocks + nsplit - 1) / nsplit > ATT_MAX_RUN) return false;
    // more than 32 blocks a CTA pay in clusters of sixteen alone, and not where a kv head has two query heads, whose P.V then keeps few
    // warps busy (three layers, split kernels against clusters, us: 16 Q / 8 KV heads, table of 4096 positions, 2000 keys, four streams
    // 192 / 213 with 35 blocks; table of 6144, 6000 keys, one stream 196 / 207 with 33)
    if (plan.cap > (C > 8 && g > 2 ? AC_CAP : 32)) return false;
    return plan.smem(g / attn_head_split(C, T, n_kv, g)) <= AC_SMEM;
}
// CTAs of the cluster that serves T tokens, 0: the split kernels do.  An SM group holds one cluster of sixteen (two where two CTAs fit
// into an SM), so they are for up to eight clusters.  Clusters of eight come in several waves above 32; they then pay where the runs are
// many enough to share out evenly (10 runs keep five CTAs of eight) and two CTAs fit into an SM, or few heads make a CTA's work short.
// Three layers, split kernels against clusters, us: 32 Q / 4 KV heads, table of 2112, 2000 keys: one stream 260 / 178, four 336 / 298,
// sixteen 710 / 629; 500 keys and a table of 640, sixteen streams 548 / 554; 32 Q / 16 KV heads, table of 640, 500 keys, sixteen streams
// 535 / 637; clusters of sixteen with four streams of those and a table of 4096: 216 / 372.
// Prompt chunks of hundreds of tokens fill the SMs either way (16 Q / 8 KV heads, 2000 tokens: 106 / 118 ms).
static int attn_cluster_size(int T, int n_kv, int g, int max_blocks, int nsplit) {
    if (T > DC_MAX_T) return 0;
    if (T * n_kv <= 8 && attn_cluster_fits(16, T, n_kv, g, max_blocks, nsplit)) return 16;
    if (!attn_cluster_fits(8, T, n_kv, g, max_blocks, nsplit)) return 0;
    if (T * n_kv <= 32) return 8;
    return nsplit >= 24 && (g <= 4 || AcPlan(8, max_blocks, nsplit).smem(g) <= 113 * 1024) ? 8 : 0;
}
bool dc_attn_cluster_ok(int T, int n_head, int n_kv, int max_blocks, int nsplit) {
    return attn_cluster_size(T, n_kv, n_head / n_kv, max_blocks, nsplit) != 0;
}

template <int C>
static int launch_attn_cluster(dc_ctx* ctx, const AttnParams& p, const dc_attn_fuse& fuse, int max_blocks) {
    const void* f = (const void*)k_attn_cluster<C>;
    const AcPlan plan(C, max_blocks, p.nsplit);
    const int g = p.n_head / p.n_kv;
    DC_TRY(dc_kernel_setup(ctx, f, AC_SMEM, "cudaFuncSetAttribute(k_attn_cluster)"));
    if (C > 8) {       // more than the portable eight, which the device has to allow
        static std::mutex mu;
        static bool done[64];
        std::lock_guard<std::mutex> lk(mu);
        const int d = ctx->device & 63;
        if (!done[d]) DC_TRY(dc_check_cuda(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "clusters of sixteen"));
        done[d] = true;
    }
    const int hs = attn_head_split(C, p.T, p.n_kv, g);
    return dc_launch_cluster(ctx, "k_attn_cluster", k_attn_cluster<C>, dim3(p.n_kv * hs * C, p.T), dim3(AC_THREADS), plan.smem(g / hs), C, p, fuse, plan.cap,
                             plan.rcap, hs);
}

size_t dc_attention_scratch_bytes(int T, int n_head, int n_kv, int max_blocks, int nsplit) {
    size_t n = 0;
    n += (size_t)T * n_head * max_blocks * DC_KV_BLOCK * 4 + 256;  // scores
    n += (size_t)T * n_head * max_blocks * 4 + 256;                // bmax
    n += (size_t)T * n_head * nsplit * 128 * 4 + 256;              // part_acc
    n += (size_t)T * n_head * nsplit * 4 + 256;                    // part_d
    n += (size_t)T * n_head * 4 + 256;                             // tickets (one per merge group)
    return n;
}

// scratch: dc_attention_scratch_bytes() bytes whose ticket area (the last
// T*n_kv ints) was zeroed once.
int dc_launch_attention(dc_ctx* ctx, const float* q, const void* k_arena, const void* v_arena,
                        const int32_t* block_tables, int max_blocks, const int32_t* seq_ids, const int32_t* positions,
                        int T, int n_head, int n_kv, float scale, int nsplit, const dc_attn_scratch* sc, float* out,
                        uint8_t* q8_out, const dc_attn_fuse* fuse) {
    const int g = n_kv > 0 ? n_head / n_kv : 0;
    if (n_kv < 1 || n_head % n_kv || g > ATT_MAX_GROUP || (g & 1))
        return dc_fail(ctx, DC_B200_UNSUPPORTED, "attention: n_head=%d n_kv=%d not supported (group must be even, <= 8)", n_head, n_kv);
    AttnParams p = {};
    p.q = q;
    p.k_arena = (const __half*)k_arena;
    p.v_arena = (const __half*)v_arena;
    p.block_tables = block_tables;
    p.max_blocks = max_blocks;
    p.seq_ids = seq_ids;
    p.positions = positions;
    p.n_head = n_head;
    p.n_kv = n_kv;
    p.T = T;
    p.nsplit = nsplit;
    p.scale = scale;
    p.scores = sc->scores;
    p.bmax = sc->bmax;
    p.part_acc = sc->part_acc;
    p.part_d = sc->part_d;
    p.tickets = sc->tickets;
    p.out = out;
    p.q8_out = q8_out;
    const int C = attn_cluster_size(T, n_kv, g, max_blocks, nsplit);
    if (C) {
        const dc_attn_fuse none = {};
        return C == 16 ? launch_attn_cluster<16>(ctx, p, fuse ? *fuse : none, max_blocks) : launch_attn_cluster<8>(ctx, p, fuse ? *fuse : none, max_blocks);
    }
    if (fuse) return dc_fail(ctx, DC_B200_UNSUPPORTED, "attention: %d blocks a sequence do not fit the fused kernel", max_blocks);
    int st = dc_launch(ctx, "k_attn_scores", k_attn_scores, dim3(nsplit, n_kv, T), dim3(128), 0, p);
    if (st != DC_B200_OK) return st;
    // runs short enough for the kernel that keeps a whole run's scores in shared memory
    if ((max_blocks + nsplit - 1) / nsplit <= ATT_MAX_RUN)
        return dc_launch(ctx, "k_attn_pv_run", k_attn_pv_run, dim3(nsplit, n_kv, T), dim3(128), 0, p);
    return dc_launch(ctx, "k_attn_pv", k_attn_pv, dim3(nsplit, n_kv, T), dim3(128), 0, p);
}

void dc_attn_scratch_bind(dc_attn_scratch* sc, uint8_t* base, int T, int n_head, int n_kv, int max_blocks, int nsplit) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        uint8_t* p = base + off;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    sc->scores = (float*)take((size_t)T * n_head * max_blocks * DC_KV_BLOCK * 4);
    sc->bmax = (float*)take((size_t)T * n_head * max_blocks * 4);
    sc->part_acc = (float*)take((size_t)T * n_head * nsplit * 128 * 4);
    sc->part_d = (float*)take((size_t)T * n_head * nsplit * 4);
    sc->tickets = (int*)take((size_t)T * n_head * 4);
}
