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
// below); a sequence table too long for a cluster's shared memory takes two kernels:
//   k_attn_scores  every run computes its scores s_t and per-block maxima;
//   k_attn_pv      every run rebuilds the reference's running-maximum chain from
//                  ALL block maxima (so its exponents are taken against exactly
//                  the reference's m_b), accumulates its blocks as the reference
//                  does, scales its partial by the product of the alphas of all
//                  later blocks, and the last run to finish (a ticket, no
//                  waiting) adds the partials and emits f32 and Q8_K output.
// Only float summation order differs from the sequential walk.
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
// global round trips between score, P.V and merge kernels.  Here the CTAs of a cluster share a sequence's blocks and exchange
// block maxima and partial sums through each other's shared memory: K and V rows of earlier positions are copied to shared memory while
// this kernel still waits for its predecessor, scores never leave the SM, and the merge reads all partials at once.
// The running-maximum chain is the reference's: a block's exponents are taken against the largest score up to that block.  What the
// reference multiplies onto its accumulator block by block (alpha) is multiplied onto the exponentials of the blocks before instead,
// within a CTA; across CTAs the partials are scaled in the merge.
// With `fuse.qkv` the kernel also norms and rotates the q heads (every CTA its own copy) and writes the new token's K and V rows
// (k_qknorm_rope_kv); the tokens of such a step belong to different sequences.
// What bounds it: the launch's dependency gap, the copy of K, one exchange of maxima and one of sums across the cluster.  32 Q / 4 KV
// heads, 2304 keys, one token: 12.5 us a layer with norm, rotation and cache write, against 29 us for the three kernels it replaces.
#define AC_THREADS 256
#define AC_CAP 32              // KV blocks a CTA holds at most (a lane each)

__device__ __forceinline__ uint32_t ac_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ac_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ac_peer(const float* mine, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 ac_peer4(const float* mine, uint32_t rank) {
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
// d = a * b + d on two floats at a time (each rounded once, as two fmaf would)
__device__ __forceinline__ void ac_fma2(float2& d, float2 a, float2 b) {
    asm("{\n.reg .b64 ra, rb, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nmov.b64 rd, {%0, %1};\n"
        "fma.rn.f32x2 rd, ra, rb, rd;\nmov.b64 {%0, %1}, rd;\n}"
        : "+f"(d.x), "+f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}
// place of the 16-byte piece i of a key's K row: eight lanes (two keys x four pieces) fall on distinct banks
__device__ __forceinline__ int ac_piece(int key, int i) { return key * 256 + ((i ^ ((key & 1) << 2)) << 4); }
__device__ __forceinline__ void ac_copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// place of (key, head) among the scores: eight heads together, eight floats more per block so that four blocks fall on distinct banks
__device__ __forceinline__ int ac_at(int key, int h) { return key * 8 + (key >> 4) * 8 + h; }

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

// C: CTAs of a cluster.  hs: clusters that share a kv head's query heads.
template <int C>
__global__ void __launch_bounds__(AC_THREADS, 2) k_attn_cluster(const AttnParams p, const dc_attn_fuse fuse, const int cap, const int hs) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* sKV = smem;                                           // K rows, after the scores V rows, after P.V partial sums: [key][256]
    float* sP = reinterpret_cast<float*>(sKV + max(cap * DC_KV_BLOCK * 256, 4 * ATT_MAX_GROUP * 128 * 4));   // scores, then weighted exponentials, see ac_at
    float* sQ = sP + cap * (DC_KV_BLOCK + 1) * 8;                  // [head][128]
    float* sPart = sQ + ATT_MAX_GROUP * 128;                       // [head][128], read by the other CTAs
    float* sBm = sPart + ATT_MAX_GROUP * 128;                      // [block][head]: block maximum, then the maximum to take exponents against
    float* sW = sBm + cap * 8;                                     // [block][head]: product of the alphas of this CTA's later blocks
    float* sMax = sW + cap * 8;                                    // [head], read by the other CTAs, as are the next two
    float* sDen = sMax + 8;
    float* sProd = sDen + 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)ac_rank(), kvh = blockIdx.x / (C * hs), part = blockIdx.x / C % hs, t = blockIdx.y, g = p.n_head / p.n_kv / hs;
    const int head0 = (kvh * hs + part) * g;                       // first of this cluster's query heads
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
    int n_blk, b0, b1;
    split_range(pos0, rank, C, n_blk, b0, b1);
    const bool early = pos0 >= 0 && b1 - b0 <= cap;
    if (early) {
        const int from = b0 * DC_KV_BLOCK, to = min(b1 * DC_KV_BLOCK, stable);
        load_k(from, from, to);
        // V's turn in the shared buffer comes after the scores; until then its rows, two lines each, come from HBM into L2
        // (a 48-layer step at 2050 keys: 0.8 % of it)
        for (int i = tid; i < 2 * (to - from); i += AC_THREADS) {
            const int key = from + (i >> 1);
            const __half* v = p.v_arena + ((size_t)table[key / DC_KV_BLOCK] * DC_KV_BLOCK + key % DC_KV_BLOCK) * row + kvh * 128 + (i & 1) * 64;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(v));
        }
    }
    auto turn_at = [&](int ps) {
        const int rp = ps < 0 ? 0 : (fuse.max_pos > 0 && ps >= fuse.max_pos) ? fuse.max_pos - 1 : ps;
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
    split_range(pos, rank, C, n_blk, b0, b1);
    const int k0 = b0 * DC_KV_BLOCK, nbl = b1 - b0, keys = max(0, min(pos + 1, b1 * DC_KV_BLOCK) - k0);
    {
        const bool same = early && pos == pos0;
        if (!same) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        load_k(k0, same ? max(k0, stable) : k0, k0 + keys - (fuse.qkv && k0 + keys == pos + 1 ? 1 : 0));
    }
    uint2 new_v = make_uint2(0u, 0u);     // the new token's V row (warp 7), which has to wait for the K rows to go
    const bool mine = fuse.qkv && keys > 0 && k0 + keys == pos + 1;
    if (fuse.qkv) {
        const float* src = fuse.qkv + (size_t)t * (p.n_head + 2 * p.n_kv) * 128;
        if (pos != pos0) turn = turn_at(pos);
        if (warp < g) reinterpret_cast<float4*>(sQ + warp * 128)[lane] = ac_norm_rope(src + (head0 + warp) * 128, fuse.qn_w != nullptr, qw, true, turn, fuse.eps, lane);
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
        for (int i = tid; i < g * 32; i += AC_THREADS) reinterpret_cast<float4*>(sQ)[i] = reinterpret_cast<const float4*>(p.q + ((size_t)t * p.n_head + head0) * 128)[i];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- scores: four lanes per pair of keys, lane `sub` takes the 16-byte pieces 4 i + sub of the rows; the queries' loads, which
    // are what this part is bound by, then serve two keys
    for (int key = 2 * (tid >> 2); key < nbl * DC_KV_BLOCK; key += AC_THREADS / 2) {
        const int sub = tid & 3;
        if (key < keys) {
            float2 kf[2][16];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) {      // (the row after the last key's is read as whatever it holds and not used)
                    const uint4 u = *reinterpret_cast<const uint4*>(sKV + ac_piece(key + k, 4 * i + sub));
                    const __half2* h2 = reinterpret_cast<const __half2*>(&u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) kf[k][4 * i + j] = __half22float2(h2[j]);
                }
            const uint32_t quad = 0xFu << (lane & ~3);
            for (int h0 = 0; h0 < g; h0 += 2) {      // g is even
                float2 d[2][2];
#pragma unroll
                for (int h = 0; h < 2; ++h) d[h][0] = d[h][1] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4* q4 = reinterpret_cast<const float4*>(sQ + (h0 + h) * 128 + (4 * i + sub) * 8);
                        const float4 a = q4[0], b = q4[1];
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            ac_fma2(d[h][k], make_float2(a.x, a.y), kf[k][4 * i]);
                            ac_fma2(d[h][k], make_float2(a.z, a.w), kf[k][4 * i + 1]);
                            ac_fma2(d[h][k], make_float2(b.x, b.y), kf[k][4 * i + 2]);
                            ac_fma2(d[h][k], make_float2(b.z, b.w), kf[k][4 * i + 3]);
                        }
                    }
                float mine = 0.0f;      // lane sub keeps (head sub / 2, key sub % 2)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        float dot = d[h][k].x + d[h][k].y;
                        dot += __shfl_xor_sync(quad, dot, 1);
                        dot += __shfl_xor_sync(quad, dot, 2);
                        if (2 * h + k == sub) mine = dot;
                    }
                const int at = key + (sub & 1);
                sP[ac_at(at, h0 + (sub >> 1))] = at < keys ? __fmul_rn(mine, p.scale) : -INFINITY;
            }
        } else {
            for (int i = sub; i < 2 * g; i += 4) sP[ac_at(key + (i & 1), i >> 1)] = -INFINITY;
        }
    }
    __syncthreads();
    // the V rows follow into the same memory while the block maxima make their way
    for (int key = tid >> 4; key < keys - (mine ? 1 : 0); key += AC_THREADS / 16) {
        const int at = k0 + key;
        const size_t off = ((size_t)table[at / DC_KV_BLOCK] * DC_KV_BLOCK + at % DC_KV_BLOCK) * row + kvh * 128 + (tid & 15) * 8;
        ac_copy16(aKV + key * 256 + (tid & 15) * 16, p.v_arena + off);
    }
    if (mine && warp == 7) *reinterpret_cast<uint2*>(sKV + (pos - k0) * 256 + 8 * lane) = new_v;
    for (int i = tid; i < nbl * 8; i += AC_THREADS) {
        const int bl = i >> 3, h = i & 7;
        if (h < g) {
            float mx = -1e30f;  // the reference's m_block starts at -1e30
#pragma unroll
            for (int k = 0; k < DC_KV_BLOCK; ++k) mx = fmaxf(mx, sP[ac_at(bl * DC_KV_BLOCK + k, h)]);
            sBm[i] = mx;
        }
    }
    __syncthreads();
    // ---- the chain: warp h, lane = block
    float incl = -1e30f, excl = -1e30f;
    if (warp < g) {
        if (lane < nbl) incl = sBm[lane * 8 + warp];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl = fmaxf(incl, u);
        }
        excl = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) excl = -1e30f;
        if (lane == 31) sMax[warp] = incl;
    }
    ac_sync();
    if (warp < g) {
        float m0 = lane < rank ? ac_peer(sMax + warp, lane) : -1e30f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
        const float m_new = fmaxf(m0, incl);
        const float alpha = lane < nbl ? fast_exp_fma(fmaxf(m0, excl) - m_new) : 1.0f;
        float after = alpha;   // inclusive product from this block on
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_down_sync(0xffffffffu, after, o);
            if (lane + o < 32) after *= u;
        }
        float later = __shfl_down_sync(0xffffffffu, after, 1);
        if (lane == 31) later = 1.0f;
        if (lane < nbl) {
            sBm[lane * 8 + warp] = m_new;
            sW[lane * 8 + warp] = later;
        }
        if (lane == 0) sProd[warp] = after;
    }
    __syncthreads();
    const int lg = g > 4 ? 3 : g > 2 ? 2 : 1;
#pragma unroll 4
    for (int i = tid; i < nbl * DC_KV_BLOCK << lg; i += AC_THREADS) {
        const int key = i >> lg, h = i & ((1 << lg) - 1), c = (key >> 4) * 8 + h;
        if (h < g) {
            const float s = sP[ac_at(key, h)];
            sP[ac_at(key, h)] = s == -INFINITY ? 0.0f : __fmul_rn(fast_exp_fma(s - sBm[c]), sW[c]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (warp < g) {
        float den = 0.0f;
        for (int key = lane; key < keys; key += 32) den += sP[ac_at(key, warp)];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        if (lane == 0) sDen[warp] = den;
    }
    // ---- P.V: four groups of threads take every fourth key, a thread two dimensions of all heads
    {
        const int kg = tid >> 6, dp = tid & 63;
        float2 a0[4], a1[4];   // head pairs, of the first and the second dimension
#pragma unroll
        for (int i = 0; i < 4; ++i) a0[i] = a1[i] = make_float2(0.0f, 0.0f);
#pragma unroll 4
        for (int key = kg; key < keys; key += 4) {
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(sKV + key * 256 + dp * 4));
            const float4* pp = reinterpret_cast<const float4*>(sP + ac_at(key, 0));
            const float4 x = pp[0], y = g > 4 ? pp[1] : x;
            const float2 vx = make_float2(v.x, v.x), vy = make_float2(v.y, v.y);
            ac_fma2(a0[0], make_float2(x.x, x.y), vx);
            ac_fma2(a1[0], make_float2(x.x, x.y), vy);
            if (g > 2) {
                ac_fma2(a0[1], make_float2(x.z, x.w), vx);
                ac_fma2(a1[1], make_float2(x.z, x.w), vy);
            }
            if (g > 4) {
                ac_fma2(a0[2], make_float2(y.x, y.y), vx);
                ac_fma2(a1[2], make_float2(y.x, y.y), vy);
            }
            if (g > 6) {
                ac_fma2(a0[3], make_float2(y.z, y.w), vx);
                ac_fma2(a1[3], make_float2(y.z, y.w), vy);
            }
        }
        __syncthreads();      // V has been read
        float* red = reinterpret_cast<float*>(sKV) + kg * ATT_MAX_GROUP * 128 + 2 * dp;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (2 * i < g) {
                *reinterpret_cast<float2*>(red + (2 * i) * 128) = make_float2(a0[i].x, a1[i].x);
                *reinterpret_cast<float2*>(red + (2 * i + 1) * 128) = make_float2(a0[i].y, a1[i].y);
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < g * 128; i += AC_THREADS) {
        const float* red = reinterpret_cast<const float*>(sKV) + i;
        sPart[i] = (red[0] + red[ATT_MAX_GROUP * 128]) + (red[2 * ATT_MAX_GROUP * 128] + red[3 * ATT_MAX_GROUP * 128]);
    }
    ac_sync();      // (also: every thread of this CTA is done with the key groups' sums)
    // ---- merge: CTA r writes the head pair r, the 256 values of one Q8_K block of the o-projection's input.  A warp takes C / 8 ranks'
    // partials, times the alphas of all ranks after; the warps' sums meet in shared memory.
    float* sSum = reinterpret_cast<float*>(sKV);                   // [warp][256], then [warp][2] denominators (the key groups' sums are done with)
    if (rank < g / 2) {
        const int head = 2 * rank + (lane >> 4), d0 = (lane & 15) * 8;
        constexpr int R = C / 8;
        float4 a[R], c[R];
        float dd[R], pr = 1.0f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            a[r] = ac_peer4(sPart + head * 128 + d0, warp * R + r);
            c[r] = ac_peer4(sPart + head * 128 + d0 + 4, warp * R + r);
            dd[r] = ac_peer(sDen + head, warp * R + r);
        }
        if ((lane & 15) < C) pr = ac_peer(sProd + head, lane & 15);            // lane of a half: the product of that rank's alphas
        float after = pr;                                                      // of this rank and all later ones
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const float u = __shfl_down_sync(0xffffffffu, after, o, 16);
            if ((lane & 15) + o < 16) after *= u;
        }
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, den = 0.0f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int next = warp * R + r + 1;
            const float suffix = __shfl_sync(0xffffffffu, after, (lane & 16) + (next & 15));
            const float f = next < C ? suffix : 1.0f;
            den += dd[r] * f;
            v[0] += a[r].x * f; v[1] += a[r].y * f; v[2] += a[r].z * f; v[3] += a[r].w * f;
            v[4] += c[r].x * f; v[5] += c[r].y * f; v[6] += c[r].z * f; v[7] += c[r].w * f;
        }
        float4* o = reinterpret_cast<float4*>(sSum + warp * 256 + lane * 8);
        o[0] = make_float4(v[0], v[1], v[2], v[3]);
        o[1] = make_float4(v[4], v[5], v[6], v[7]);
        if ((lane & 15) == 0) sSum[8 * 256 + warp * 2 + (lane >> 4)] = den;
    }
    __syncthreads();
    if (rank < g / 2 && warp == 0) {
        const int head = 2 * rank + (lane >> 4), d0 = (lane & 15) * 8;
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, den = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const float4* o = reinterpret_cast<const float4*>(sSum + w * 256 + lane * 8);
            const float4 x = o[0], y = o[1];
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
            v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
            den += sSum[8 * 256 + w * 2 + (lane >> 4)];
        }
        const float inv = (den > 0.0f && isfinite(den)) ? __fdiv_rn(1.0f, __fadd_rn(den, 1e-6f)) : 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= inv;
        if (p.out) {
            float* o = p.out + ((size_t)t * p.n_head + head0 + head) * 128 + d0;
            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
        if (p.q8_out) quantize_block_q8f_regs(v, p.q8_out + ((size_t)t * (p.n_head / 2) + head0 / 2 + rank) * DC_Q8F_BYTES, lane);
    }
    ac_sync();      // nobody leaves while its shared memory is read
}

static size_t attn_cluster_smem(int cap) {
    const size_t k = (size_t)cap * DC_KV_BLOCK * 256, red = 4 * ATT_MAX_GROUP * 128 * 4;
    return (k > red ? k : red) + ((size_t)cap * (DC_KV_BLOCK + 1) * 8 + 2 * ATT_MAX_GROUP * 128 + (size_t)cap * 16 + 24) * 4;
}
bool dc_attn_cluster_ok(int max_blocks) { return max_blocks <= 16 * AC_CAP; }

template <int C>
static int launch_attn_cluster(dc_ctx* ctx, const AttnParams& p, const dc_attn_fuse& fuse, int max_blocks) {
    const void* f = (const void*)k_attn_cluster<C>;
    const int cap = (max_blocks + C - 1) / C, g = p.n_head / p.n_kv;
    const size_t smem = attn_cluster_smem(cap);
    DC_TRY(dc_kernel_setup(ctx, f, (int)attn_cluster_smem(AC_CAP), "cudaFuncSetAttribute(k_attn_cluster)"));
    if (C > 8) {       // more than the portable eight, which the device has to allow
        static std::mutex mu;
        static bool done[64];
        std::lock_guard<std::mutex> lk(mu);
        const int d = ctx->device & 63;
        if (!done[d]) DC_TRY(dc_check_cuda(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "clusters of sixteen"));
        done[d] = true;
    }
    // few tokens: two clusters share a kv head's query heads, as long as there is an SM for every CTA
    const int hs = g % 4 == 0 && 2 * p.T * p.n_kv * C <= 128 ? 2 : 1;
    return dc_launch_cluster(ctx, "k_attn_cluster", k_attn_cluster<C>, dim3(p.n_kv * hs * C, p.T), dim3(AC_THREADS), smem, C, p, fuse, cap, hs);
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
    // The cluster's shared memory holds all keys of a sequence up to a length; longer ones take the split kernels.  Clusters of sixteen
    // halve a CTA's share but only one fits into a group of SMs: they pay for up to eight clusters, or where eight CTAs cannot hold the keys
    // (16 Q / 8 KV heads, 512 keys, 4 tokens: 11 us a launch with eight, 26 us with sixteen).
    if (dc_attn_cluster_ok(max_blocks)) {
        const dc_attn_fuse none = {};
        if (max_blocks > 8 * AC_CAP || T * n_kv <= 8) return launch_attn_cluster<16>(ctx, p, fuse ? *fuse : none, max_blocks);
        return launch_attn_cluster<8>(ctx, p, fuse ? *fuse : none, max_blocks);
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
