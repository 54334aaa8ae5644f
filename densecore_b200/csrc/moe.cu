// Fused MoE layer (MUL_MAT_ID).  Replaces cb_moe_forward
// (core/src/llm/moe/exec.cpp:813) -> RouteMoESoftmaxTopK (:734) ->
// CpuBackend::ForwardMoE (core/src/backend/cpu_backend_moe_ops.cpp:1195):
//   k_router      router logits (F32 matmul, core/src/llm/graph/decoder.cpp:2265),
//                 stable top-k + weights (core/src/llm/moe/native.cpp:610-676),
//                 token->expert bucketing (core/src/moe/moe_routing.cpp:534-603)
//   k_moe_rows<PAIR> gate/up + SwiGLU for every (distinct expert, row), each expert's
//                 weights read once for all its tokens (native.cpp:3929-4345)
//   k_moe_rows    down projection per assignment (native.cpp:3051-3295)
//   k_moe_combine weighted sum in the reference's order
//                 (cpu_backend_moe_ops.cpp:1578-1597, moe_routing.cpp:647-676)
#include "dc_common.cuh"
#include "dc_internal.h"
#include "dc_launch.cuh"
#include "dc_rows.cuh"

using namespace dc;

#define MOE_MAX_E 256
#define MOE_MAX_K 16

// ------------------------------------------------------------------ router
struct RouterParams {
    const float* wr;      // [E][H] f32
    const float* xn;      // [T][H] f32 (normed hidden state)
    int E, H, T, top_k;
    float scale;          // moe_routed_scaling_factor
    int mode;             // DC_ROUTE_STABLE (top-k on logits) or DC_ROUTE_SOFTMAX (softmax over all experts first)
    int ep_lo, ep_hi;     // experts owned by this GPU
    float* logits;        // [T][E]
    int32_t* ids;         // [T][top_k]
    float* weights;       // [T][top_k]
    int* ticket;          // zero-initialised, self-resetting
    int* n_active;        // U
    int32_t* uexp;        // distinct local experts, ascending, once for every DC_MOE_PASS of their tokens
    int32_t* uoff;        // their offsets into uassign, and the end
    int32_t* uassign;     // [T*top_k] assignment indices t*top_k+k, grouped by expert, routing order inside
    dc_route_norm norm;   // x given: rows still to be normed
    bool sixteenths;      // one token: its logits as sixteen partial sums in order, as the persistent kernel forms them
};

__device__ __forceinline__ unsigned long long route_key(float v, int id) {
    uint32_t u;
    if (v != v) u = 0u;
    else {
        if (v == 0.0f) v = 0.0f;  // -0 == +0 for the comparator
        u = __float_as_uint(v);
        u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    }
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)id);
}

// expf rounded as the host library rounds it: the double-precision exponential (1 ulp of double) rounded once
// to float is the correctly rounded float result except on a 2^-29 sliver of arguments, and so is glibc's expf.
// The generic router compares probabilities for equality (ties go to the lower expert id), so its
// exponentials must be the CPU's bit for bit.
__device__ __forceinline__ float expf_cr(float x) { return (float)exp((double)x); }

// Routing of token t by one warp: stable top-k on the logits (native router) or on the softmax probabilities
// (generic router), then the routing weights.  s_prob: MOE_MAX_E floats of shared memory owned by this warp;
// s_ids (optional): shared copy of the ids for the bucketing that follows in k_router.
__device__ __forceinline__ void route_token(const RouterParams& p, int t, int lane, float* s_prob, int32_t* s_ids) {
    float lv[MOE_MAX_E / 32];
    bool taken[MOE_MAX_E / 32];
#pragma unroll
    for (int j = 0; j < MOE_MAX_E / 32; ++j) {
        const int id = j * 32 + lane;
        lv[j] = id < p.E ? __ldcg(p.logits + (size_t)t * p.E + id) : 0.0f;
        taken[j] = id >= p.E;
    }
    if (p.mode == DC_ROUTE_SOFTMAX) {
        // softmax over all experts: expf(x - max), sum in index order, times 1/sum
        // (core/include/densecore/simd/simd_ops.h:1171-1195); selection then runs on the probabilities
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < MOE_MAX_E / 32; ++j)
            if (!taken[j]) mx = fmaxf(mx, lv[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
        for (int j = 0; j < MOE_MAX_E / 32; ++j) {
            if (!taken[j]) {
                lv[j] = expf_cr(__fsub_rn(lv[j], mx));
                s_prob[j * 32 + lane] = lv[j];
            }
        }
        __syncwarp();
        float sum = 0.0f;
        if (lane == 0)
            for (int e = 0; e < p.E; ++e) sum = __fadd_rn(sum, s_prob[e]);
        sum = __shfl_sync(0xffffffffu, sum, 0);
        const float inv = __fdiv_rn(1.0f, sum);
#pragma unroll
        for (int j = 0; j < MOE_MAX_E / 32; ++j)
            if (!taken[j]) lv[j] = __fmul_rn(lv[j], inv);
        __syncwarp();
    }
    float sel_l[MOE_MAX_K];
    for (int k = 0; k < p.top_k; ++k) {
        unsigned long long best = 0ull;
#pragma unroll
        for (int j = 0; j < MOE_MAX_E / 32; ++j) {
            if (!taken[j]) {
                const unsigned long long key = route_key(lv[j], j * 32 + lane);
                best = key > best ? key : best;
            }
        }
        // a real candidate's key is never 0 (its low word is 0xFFFFFFFF - id), so 0 means "none"
        unsigned long long win = best;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ok = __shfl_xor_sync(0xffffffffu, win, o);
            win = ok > win ? ok : win;
        }
        const int wid = (int)(0xFFFFFFFFu - (uint32_t)(win & 0xFFFFFFFFull));
#pragma unroll
        for (int j = 0; j < MOE_MAX_E / 32; ++j)
            if (j * 32 + lane == wid) taken[j] = true;
        // the winner's value back out of its key (NaN stays NaN; -0 was made +0, which exp treats alike):
        // no load per round
        const uint32_t ku = (uint32_t)(win >> 32);
        const float wl = __uint_as_float((ku & 0x80000000u) ? (ku & 0x7FFFFFFFu) : ~ku);
        if (k < MOE_MAX_K) sel_l[k] = wl;
        if (lane == 0) {
            p.ids[t * p.top_k + k] = wid;
            if (s_ids) s_ids[t * p.top_k + k] = wid;
        }
    }
    if (lane == 0 && p.mode == DC_ROUTE_SOFTMAX) {
        // renormalise over the picks in pick order: w * (1 / sum) (core/src/moe/moe_routing.cpp:90-101),
        // then the routed scaling factor (core/src/llm/moe/exec.cpp:764-768)
        float sum = 0.0f;
        for (int k = 0; k < p.top_k; ++k) sum = __fadd_rn(sum, sel_l[k]);
        const float is = sum > 0.0f ? __fdiv_rn(1.0f, sum) : 1.0f;
        for (int k = 0; k < p.top_k; ++k)
            p.weights[t * p.top_k + k] = __fmul_rn(sum > 0.0f ? __fmul_rn(sel_l[k], is) : sel_l[k], p.scale);
    } else if (lane == 0) {
        // weights over the selected experts only (native.cpp:649-674)
        float mx = -INFINITY;
        bool finite = true;
        for (int k = 0; k < p.top_k; ++k) {
            finite = finite && isfinite(sel_l[k]);
            if (isfinite(sel_l[k]) && sel_l[k] > mx) mx = sel_l[k];
        }
        float den = 0.0f, wv[MOE_MAX_K];
        if (finite && isfinite(mx)) {
            for (int k = 0; k < p.top_k; ++k) {
                wv[k] = expf(sel_l[k] - mx);
                den += wv[k];
            }
        }
        const bool ok = den > 0.0f && isfinite(den);
        for (int k = 0; k < p.top_k; ++k) {
            const float w = ok ? __fdiv_rn(wv[k], den) : __fdiv_rn(1.0f, (float)p.top_k);
            p.weights[t * p.top_k + k] = __fmul_rn(w, p.scale);
        }
    }
}

// Routing of token t by one warp (DC_ROUTE_STABLE): the best expert left is found by two warp-wide reductions, of the 32-bit keys and, among
// equal ones, of the ids; the weights are those of the persistent kernel (exponentials side by side, their sum in pick order).
// Bound by the chain of top_k rounds.  Expert layers of 2048 columns, us at 3 / 12 tokens: 128 experts of 768 columns, 8 picks 70 / 148;
// 256 experts of 512 65 / 135.  One CTA that compared every expert with every other, a token after the other, made these 79 / 173 and
// 82 / 203, and route_token's rounds of 64-bit exchanges were 5 us a launch where these are 2.
__device__ __forceinline__ void route_token_stable(const RouterParams& p, int t, int lane, int32_t* s_ids) {
    uint32_t key[MOE_MAX_E / 32];      // order of the logits, from 1 (NaN) on; 0: none left
#pragma unroll
    for (int j = 0; j < MOE_MAX_E / 32; ++j) {
        const int e = j * 32 + lane;
        key[j] = e < p.E ? (uint32_t)(route_key(__ldcg(p.logits + (size_t)t * p.E + e), e) >> 32) + 1u : 0u;
    }
    int pick = 0;
    uint32_t at = 0u;      // lane k: the k-th pick and its key
#pragma unroll 1
    for (int k = 0; k < p.top_k; ++k) {
        uint32_t best = key[0];
        int id = lane;
#pragma unroll
        for (int j = 1; j < MOE_MAX_E / 32; ++j)
            if (key[j] > best) {      // (equal: the lower id stays)
                best = key[j];
                id = j * 32 + lane;
            }
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        const int win = (int)__reduce_min_sync(0xffffffffu, best == top ? (uint32_t)id : 0xffffffffu);
#pragma unroll
        for (int j = 0; j < MOE_MAX_E / 32; ++j)
            if (j * 32 + lane == win) key[j] = 0u;
        if (lane == k) {
            pick = win;
            at = top - 1u;
        }
    }
    const bool own = lane < p.top_k;
    const float v = own ? __uint_as_float((at & 0x80000000u) ? (at & 0x7FFFFFFFu) : ~at) : -INFINITY;     // the logit (-0 became +0)
    // weights over the selected experts only (native.cpp:649-674)
    const bool finite = __all_sync(0xffffffffu, !own || isfinite(v));
    float mx = own && isfinite(v) ? v : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float ev = finite && isfinite(mx) && own ? expf(v - mx) : 0.0f;
    float den = 0.0f;
#pragma unroll 1
    for (int k = 0; k < p.top_k; ++k) den += __shfl_sync(0xffffffffu, ev, k);
    if (own) {
        const bool ok = den > 0.0f && isfinite(den);
        const int i = t * p.top_k + lane;
        p.weights[i] = __fmul_rn(ok ? __fdiv_rn(ev, den) : __fdiv_rn(1.0f, (float)p.top_k), p.scale);
        p.ids[i] = pick;
        s_ids[i] = pick;
    }
}

__global__ void __launch_bounds__(256) k_router(const RouterParams p) {
    __shared__ int s_last;
    __shared__ float s_prob[8][MOE_MAX_E];
    __shared__ __align__(16) int32_t s_ids[DC_MAX_T * MOE_MAX_K + 4];
    __shared__ int s_wsum_a[8], s_wsum_c[8];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // logits: two experts per CTA, four warps per expert, each warp a quarter of the row
    // with all of its loads issued before the first use.  The router weights do not depend on the
    // previous kernel: the first batch is fetched while this kernel still waits for it.
    float4 wv0[4];
    {
        const int e = blockIdx.x * 2 + (warp >> 2), quarter = warp & 3, seg = p.H / 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = j * 32 + lane;
            wv0[j] = (p.wr && e < p.E && i < seg / 4)
                         ? reinterpret_cast<const float4*>(p.wr + (size_t)e * p.H + quarter * seg)[i]
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    float4 nw[2] = {};      // norm weights, which are older than the previous kernel too
    if (p.norm.x) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if ((int)threadIdx.x + 256 * j < p.H / 4) nw[j] = reinterpret_cast<const float4*>(p.norm.w)[threadIdx.x + 256 * j];
    }
    pdl_wait();
    const float* xn = p.xn;
    if (p.norm.x) {
        // every CTA norms all rows (k_rmsnorm_q8k's arithmetic) into shared memory; the blocks to quantise are shared out
        extern __shared__ __align__(16) float s_xn[];
        __shared__ double s_ss[8][4];
        float4* sx4 = reinterpret_cast<float4*>(s_xn);
        const int n4 = p.H / 4;
        for (int t = 0; t < p.T; ++t) {
            const float4* xr = reinterpret_cast<const float4*>(p.norm.x + (size_t)t * p.H);
            double ss = 0.0;
            for (int i0 = 0; i0 < n4; i0 += 512) {       // two loads in flight
                const int i = i0 + threadIdx.x, k = i + 256;
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), a = i < n4 ? __ldcg(xr + i) : zero, b = k < n4 ? __ldcg(xr + k) : zero;
                if (i < n4) sx4[t * n4 + i] = a;
                if (k < n4) sx4[t * n4 + k] = b;
                ss += ((double)a.x * a.x + (double)a.y * a.y) + ((double)a.z * a.z + (double)a.w * a.w);
                ss += ((double)b.x * b.x + (double)b.y * b.y) + ((double)b.z * b.z + (double)b.w * b.w);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) s_ss[warp][t] = ss;
        }
        __syncthreads();
        for (int t = 0; t < p.T; ++t) {
            double tot = 0.0;
#pragma unroll
            for (int i = 0; i < 8; ++i) tot += s_ss[i][t];
            const float mean = (float)(tot / (double)p.H);
            const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, p.norm.eps)));
            for (int i = threadIdx.x, j = 0; i < n4; i += 256, ++j) {
                const float4 v = sx4[t * n4 + i], w = j < 2 ? nw[j] : reinterpret_cast<const float4*>(p.norm.w)[i];
                sx4[t * n4 + i] = make_float4(__fmul_rn(__fmul_rn(v.x, scale), w.x), __fmul_rn(__fmul_rn(v.y, scale), w.y),
                                              __fmul_rn(__fmul_rn(v.z, scale), w.z), __fmul_rn(__fmul_rn(v.w, scale), w.w));
            }
        }
        __syncthreads();
        xn = s_xn;
    }
    if (p.wr) {
        __shared__ float s_part[8][DC_MAX_T];
        const int e = blockIdx.x * 2 + (warp >> 2), quarter = warp & 3;
        const int seg = p.H / 4;  // H is a multiple of 256
        float acc[DC_MAX_T];
#pragma unroll
        for (int t = 0; t < DC_MAX_T; ++t) acc[t] = 0.0f;
        if (p.sixteenths) {
            if (e < p.E) {
                const int n4 = seg / 16;      // float4s of a sixteenth
                const float4* w4 = reinterpret_cast<const float4*>(p.wr + (size_t)e * p.H + quarter * seg);
                const float4* x4 = reinterpret_cast<const float4*>(xn + quarter * seg);
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    for (int i = lane; i < n4; i += 32) {
                        const float4 w = n4 == 32 ? wv0[s] : w4[s * n4 + i], x = x4[s * n4 + i];
                        acc[s] = fmaf(w.x, x.x, acc[s]);
                        acc[s] = fmaf(w.y, x.y, acc[s]);
                        acc[s] = fmaf(w.z, x.z, acc[s]);
                        acc[s] = fmaf(w.w, x.w, acc[s]);
                    }
            }
        } else if (e < p.E) {
            const float4* w4 = reinterpret_cast<const float4*>(p.wr + (size_t)e * p.H + quarter * seg);
            for (int i0 = 0; i0 < seg / 4; i0 += 128) {
                float4 wv[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = i0 + j * 32 + lane;
                    wv[j] = i0 == 0 ? wv0[j] : (i < seg / 4 ? w4[i] : make_float4(0.f, 0.f, 0.f, 0.f));
                }
#pragma unroll
                for (int t = 0; t < DC_MAX_T; ++t) {
                    if (t < p.T) {
                        const float4* x4 = reinterpret_cast<const float4*>(xn + (size_t)t * p.H + quarter * seg);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int i = i0 + j * 32 + lane;
                            if (i < seg / 4) {
                                const float4 xv = x4[i];
                                acc[t] = fmaf(wv[j].x, xv.x, acc[t]);
                                acc[t] = fmaf(wv[j].y, xv.y, acc[t]);
                                acc[t] = fmaf(wv[j].z, xv.z, acc[t]);
                                acc[t] = fmaf(wv[j].w, xv.w, acc[t]);
                            }
                        }
                    }
                }
            }
        }
        const int sums = p.sixteenths ? 4 : p.T;
#pragma unroll
        for (int t = 0; t < DC_MAX_T; ++t) {
            if (t < sums) {
                float v = acc[t];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) s_part[warp][t] = v;
            }
        }
        __syncthreads();
        if (p.sixteenths) {
            const int which = threadIdx.x, ee = blockIdx.x * 2 + which;
            if (which < 2 && ee < p.E) {
                float v = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) v += s_part[which * 4 + i / 4][i % 4];
                p.logits[ee] = v;
            }
        } else if (threadIdx.x < 2 * p.T) {
            const int which = threadIdx.x / p.T, t = threadIdx.x % p.T, ee = blockIdx.x * 2 + which;
            if (ee < p.E)
                p.logits[(size_t)t * p.E + ee] = (s_part[which * 4][t] + s_part[which * 4 + 1][t]) +
                                                 (s_part[which * 4 + 2][t] + s_part[which * 4 + 3][t]);
        }
    }
    // release: the CTA barrier puts this CTA's logits before thread 0's ticket, whose release half publishes them;
    // acquire: the last CTA's thread 0 sees the others' logits through the ticket's acquire half, and the CTA
    // barrier passes that on
    __syncthreads();
    if (threadIdx.x == 0) {
        int old;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p.ticket), "r"(1) : "memory");
        s_last = old == (int)gridDim.x - 1;
        if (s_last) *p.ticket = 0;
    }
    if (p.norm.x) {      // off the chain that the picks wait for
        const int nb = p.H / DC_QK_K;
        for (int i = warp * gridDim.x + blockIdx.x; i < p.T * nb; i += 8 * gridDim.x)
            quantize_block_q8k_warp<true>(xn + i * DC_QK_K, p.norm.q8_out + (size_t)i * DC_Q8F_BYTES, lane);
    }
    __syncthreads();
    if (!s_last) return;

    // ---- top-k per token, one warp per token
    if (threadIdx.x < 4) s_ids[p.T * p.top_k + threadIdx.x] = -1;
    for (int t = warp; t < p.T; t += 8) {
        if (p.mode == DC_ROUTE_STABLE) route_token_stable(p, t, lane, s_ids);
        else route_token(p, t, lane, s_prob[warp], s_ids);
    }
    __syncthreads();
    if (p.T == 1) {      // every pick is an expert's only token: the picks of this GPU's experts by ascending id
        if (threadIdx.x < 32) {
            const int k = threadIdx.x, own = k < p.top_k ? s_ids[k] : -1;
            const bool local = own >= p.ep_lo && own < p.ep_hi;
            int at = 0;
            for (int j = 0; j < p.top_k; ++j) at += s_ids[j] >= p.ep_lo && s_ids[j] < own;
            if (local) {
                p.uexp[at] = own;
                p.uoff[at] = at;
                p.uassign[at] = k;
            }
            const int n = __popc(__ballot_sync(0xffffffffu, local));
            if (k == 0) {
                *p.n_active = n;
                p.uoff[n] = n;
            }
        }
        return;
    }
    // ---- bucketing: thread e owns expert e
    const int A = p.T * p.top_k;
    const int me = threadIdx.x;
    int cnt = 0;
    if (me < p.E && me >= p.ep_lo && me < p.ep_hi)
        for (int i = 0; i < A; i += 4) {      // (s_ids is padded with -1)
            const int4 x = *reinterpret_cast<const int4*>(s_ids + i);
            cnt += (x.x == me) + (x.y == me) + (x.z == me) + (x.w == me);
        }
    int act = (cnt + DC_MOE_PASS - 1) / DC_MOE_PASS;
    // inclusive scans of (act, cnt) over the 256 threads
    int sa = act, scn = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a2 = __shfl_up_sync(0xffffffffu, sa, o), c2 = __shfl_up_sync(0xffffffffu, scn, o);
        if (lane >= o) {
            sa += a2;
            scn += c2;
        }
    }
    if (lane == 31) {
        s_wsum_a[warp] = sa;
        s_wsum_c[warp] = scn;
    }
    __syncthreads();
    int base_a = 0, base_c = 0, tot_a = 0, tot_c = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) {
            base_a += s_wsum_a[w];
            base_c += s_wsum_c[w];
        }
        tot_a += s_wsum_a[w];
        tot_c += s_wsum_c[w];
    }
    if (act) {
        const int u = base_a + sa - act, off = base_c + scn - cnt;
        for (int i = 0; i < act; ++i) {
            p.uexp[u + i] = me;
            p.uoff[u + i] = off + DC_MOE_PASS * i;
        }
        int o = off;
        for (int i = 0; o < off + cnt; i += 4) {
            const int4 x = *reinterpret_cast<const int4*>(s_ids + i);
            if (x.x == me) p.uassign[o++] = i;
            if (x.y == me) p.uassign[o++] = i + 1;
            if (x.z == me) p.uassign[o++] = i + 2;
            if (x.w == me) p.uassign[o++] = i + 3;
        }
    }
    if (threadIdx.x == 0) {
        *p.n_active = tot_a;
        p.uoff[tot_a] = tot_c;
    }
}

// ------------------------------------------- router over a prompt chunk
// The same arithmetic as k_router for any number of tokens, bit for bit: four warps per expert, a quarter of the row each, lane partials
// chained by fma in the same element order, butterfly sum, quarters added pairwise.  A warp keeps the partials of four experts x eight
// tokens, so that twelve 16-byte loads feed 128 multiply-adds (the first form, two experts x sixteen tokens a CTA with one expert a warp,
// read every token's row 64 times over: 194 us for 2048 tokens, 128 experts and 2048 columns, at 5 % of the multiply-adds' rate).
// Its 32 sums over the lanes take 31 exchanges: each step halves the sums that a lane still holds, and adds the same pairs
// as a butterfly of every sum would.  No bucketing: the chunk's assignments are grouped by k_moe_group.
#define RB_E 4     // experts of a warp
#define RB_T 8     // tokens of a warp
__global__ void __launch_bounds__(256) k_router_logits_batched(const RouterParams p) {
    __shared__ float s_part[8][RB_E * RB_T];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3, seg = p.H / 4;
    const int e0 = (blockIdx.x * 2 + (warp >> 2)) * RB_E, t0 = blockIdx.y * RB_T;
    float acc[RB_E * RB_T];
#pragma unroll
    for (int i = 0; i < RB_E * RB_T; ++i) acc[i] = 0.0f;
    const float4 *w4[RB_E], *x4[RB_T];   // (experts and tokens past the end are read as the last one)
#pragma unroll
    for (int e = 0; e < RB_E; ++e) w4[e] = reinterpret_cast<const float4*>(p.wr + (size_t)min(e0 + e, p.E - 1) * p.H + quarter * seg);
#pragma unroll
    for (int t = 0; t < RB_T; ++t) x4[t] = reinterpret_cast<const float4*>(p.xn + (size_t)min(t0 + t, p.T - 1) * p.H + quarter * seg);
    for (int i = lane; i < seg / 4; i += 32) {
        float4 w[RB_E], x[RB_T];
#pragma unroll
        for (int e = 0; e < RB_E; ++e) w[e] = w4[e][i];
#pragma unroll
        for (int t = 0; t < RB_T; ++t) x[t] = x4[t][i];
#pragma unroll
        for (int e = 0; e < RB_E; ++e)
#pragma unroll
            for (int t = 0; t < RB_T; ++t) {
                float& a = acc[e * RB_T + t];
                a = fmaf(w[e].x, x[t].x, a);
                a = fmaf(w[e].y, x[t].y, a);
                a = fmaf(w[e].z, x[t].z, a);
                a = fmaf(w[e].w, x[t].w, a);
            }
    }
    // after the step over lane bit o a lane holds the sums whose index has that bit as its own lane number has
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float mine = upper ? acc[i + o] : acc[i], other = upper ? acc[i] : acc[i + o];
            acc[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
        }
    }
    s_part[warp][lane] = acc[0];
    __syncthreads();
    if (threadIdx.x < 2 * RB_E * RB_T) {
        const int which = threadIdx.x >> 5, i = threadIdx.x & 31;
        const int e = (blockIdx.x * 2 + which) * RB_E + i / RB_T, t = t0 + i % RB_T;
        if (e < p.E && t < p.T)
            p.logits[(size_t)t * p.E + e] = (s_part[which * 4][i] + s_part[which * 4 + 1][i]) + (s_part[which * 4 + 2][i] + s_part[which * 4 + 3][i]);
    }
}

__global__ void __launch_bounds__(256) k_router_select_batched(const RouterParams p) {
    __shared__ float s_prob[8][MOE_MAX_E];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 8 + warp;
    if (t < p.T) route_token(p, t, lane, s_prob[warp], nullptr);
}

// Router of a prompt chunk: logits [T][E], ids and weights [T][top_k] for any T.
int dc_launch_router_batched(dc_ctx* ctx, const dc_weight* wr, const float* xn, int T, int top_k, float scale, float* logits,
                             int32_t* ids, float* weights, int mode) {
    if (!wr || wr->type != DC_TYPE_F32) return dc_fail(ctx, DC_B200_UNSUPPORTED, "router weight must be F32");
    const int E = (int)wr->N;
    if (E < 1 || E > MOE_MAX_E || top_k < 1 || top_k > MOE_MAX_K || top_k > E || T < 1)
        return dc_fail(ctx, DC_B200_UNSUPPORTED, "router: E=%d top_k=%d T=%d out of range", E, top_k, T);
    RouterParams p = {};
    p.wr = (const float*)wr->dev;
    p.xn = xn;
    p.E = E;
    p.H = (int)wr->K;
    p.T = T;
    p.top_k = top_k;
    p.scale = scale;
    p.mode = mode;
    p.ep_lo = 0;
    p.ep_hi = E;
    p.logits = logits;
    p.ids = ids;
    p.weights = weights;
    k_router_logits_batched<<<dim3((E + 2 * RB_E - 1) / (2 * RB_E), (T + RB_T - 1) / RB_T), 256, 0, ctx->stream>>>(p);
    {
        const int st = dc_check_cuda(ctx, cudaGetLastError(), "k_router_logits_batched");
        if (st != DC_B200_OK) return st;
    }
    k_router_select_batched<<<(T + 7) / 8, 256, 0, ctx->stream>>>(p);
    return dc_check_cuda(ctx, cudaGetLastError(), "k_router_select_batched");
}

// --------------------------------------------------- expert matmul kernel
// Down projection (PAIR false): the routing was final before this kernel could start (the gate/up kernel lets its successor start only
// after its own wait, and so does the quantiser between the two, an ordinary launch), so the expert rows can be requested while this
// kernel still waits for its predecessor's output.  Gate/up: the expert ids come from the router kernel just before.
template <int TYPE, int NP, bool ONE, bool ALONE, bool PAIR>
__global__ void __launch_bounds__(RW_THREADS, TYPE == DC_TYPE_Q4_K ? 3 : 2) k_moe_rows(const RowsParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    rows_cta<TYPE, NP, ONE, ALONE, true, PAIR, false, !PAIR>(p, smem, blockIdx.x, gridDim.x, 0, 0);
}

template <int TYPE, int NP, bool ONE, bool PAIR, bool ALONE>
static int launch_moe_rows_as(dc_ctx* ctx, const RowsParams& p, size_t smem, int max_tiles) {
    const void* f = (const void*)k_moe_rows<TYPE, NP, ONE, ALONE, PAIR>;
    int st = dc_kernel_setup(ctx, f, 220 * 1024, "cudaFuncSetAttribute(k_moe_rows)");
    if (st != DC_B200_OK) return st;
    int per_sm = dc_kernel_occupancy(ctx, f, RW_THREADS, smem);
    if (per_sm < 1) per_sm = 1;
    const int groups = RW_WARPS / p.S, useful = (max_tiles + groups - 1) / groups;
    const int grid = useful < ctx->num_sms * per_sm ? useful : ctx->num_sms * per_sm;
    return dc_launch(ctx, "k_moe_rows", k_moe_rows<TYPE, NP, ONE, ALONE, PAIR>, dim3(grid), dim3(RW_THREADS), smem, p);
}
template <int TYPE, int NP, bool ONE, bool PAIR>
static int launch_moe_rows(dc_ctx* ctx, const RowsParams& p, size_t smem, int max_tiles) {
    return p.S == 1 ? launch_moe_rows_as<TYPE, NP, ONE, PAIR, true>(ctx, p, smem, max_tiles) : launch_moe_rows_as<TYPE, NP, ONE, PAIR, false>(ctx, p, smem, max_tiles);
}
template <int TYPE, bool PAIR>
static int launch_moe_rows_np(dc_ctx* ctx, const RowsParams& p, int np, size_t smem, int max_tiles) {
    if (p.T == 1) return launch_moe_rows<TYPE, 1, true, PAIR>(ctx, p, smem, max_tiles);
    if (np == 1) return launch_moe_rows<TYPE, 1, false, PAIR>(ctx, p, smem, max_tiles);
    return launch_moe_rows<TYPE, 2, false, PAIR>(ctx, p, smem, max_tiles);
}

// w0/w1: expert tensors [K, N, E].  pair: gate/up + SwiGLU, activations are the T
// token rows; else down, activations are the T*top_k assignment rows.
int dc_launch_moe_mm(dc_ctx* ctx, bool pair, const dc_weight* w0, const dc_weight* w1, const uint8_t* act_q8,
                     int T, int top_k, int e_base, const dc_moe_route* rt, float* out, const float* act_f32) {
    RowsParams p = {};
    p.w0 = w0->dev;
    p.w1 = pair ? w1->dev : nullptr;
    p.e_base = e_base;
    p.type = w0->type;
    p.row_bytes = (int)w0->row_bytes;
    p.N = (int)w0->N;
    p.K = (int)w0->K;
    p.nb = p.K / DC_QK_K;
    if (p.type != DC_TYPE_Q4_K && p.type != DC_TYPE_Q6_K)
        return dc_fail(ctx, DC_B200_UNSUPPORTED, "moe: expert weight type %d is not Q4_K/Q6_K", p.type);
    if (pair && (w1->type != w0->type || w1->N != w0->N || w1->K != w0->K))
        return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "moe: gate and up tensors differ in type or shape");
    p.act_q8 = act_q8;
    p.act_f32 = act_f32;
    p.T = T;
    p.top_k = top_k;
    p.n_active = rt->n_active;
    p.uexp = rt->uexp;
    p.uoff = rt->uoff;
    p.uassign = rt->uassign;
    p.out = out;
    // A kernel takes up to DC_MOE_PASS tokens of an expert; the few experts with more come several times over and are read again from
    // L2.  (Kernels for sixteen tokens an expert hold 255 registers, eight warps an SM: 259 us for 16 tokens of 8 out of 128 experts.)
    // act_rows: the passes that one CTA's neighbouring tiles touch are one more than its share of them, rounded up (a pass has 16 tiles at
    // least, N being a multiple of 256, and a CTA eight or fewer where the SMs are not full).
    const int A = T * top_k, E = (int)w0->E, most = E + A / DC_MOE_PASS, U = most < A ? most : A;
    const int span = U <= 1 ? 1 : (U + ctx->num_sms - 1) / ctx->num_sms + 1, per = T < DC_MOE_PASS ? T : DC_MOE_PASS;
    p.act_rows = span * per < A ? span * per : A;
    p.tiles = (p.N + 15) / 16;
    const int np = T <= 2 ? 1 : 2, all = U * p.tiles;
    const size_t smem = rows_plan(p, np, p.type == DC_TYPE_Q6_K, all, ctx->num_sms);
    if (!smem) return dc_fail(ctx, DC_B200_UNSUPPORTED, "moe: K=%d needs too much shared memory for %d tokens", p.K, T);
    if (p.type == DC_TYPE_Q4_K) return pair ? launch_moe_rows_np<DC_TYPE_Q4_K, true>(ctx, p, np, smem, all) : launch_moe_rows_np<DC_TYPE_Q4_K, false>(ctx, p, np, smem, all);
    return pair ? launch_moe_rows_np<DC_TYPE_Q6_K, true>(ctx, p, np, smem, all) : launch_moe_rows_np<DC_TYPE_Q6_K, false>(ctx, p, np, smem, all);
}

int dc_launch_router(dc_ctx* ctx, const dc_weight* wr, const float* xn, int n_expert, int T, int top_k, float scale,
                     int ep_lo, int ep_hi, const dc_moe_route* rt, int mode, const dc_route_norm* norm, bool sixteenths) {
    // wr == nullptr: rt->logits already holds the router logits (routing only)
    if (wr && wr->type != DC_TYPE_F32) return dc_fail(ctx, DC_B200_UNSUPPORTED, "router weight must be F32");
    const int E = wr ? (int)wr->N : n_expert;
    if (E < 1 || E > MOE_MAX_E || top_k < 1 || top_k > MOE_MAX_K || top_k > E || T < 1 || T > DC_MAX_T)
        return dc_fail(ctx, DC_B200_UNSUPPORTED, "router: E=%d top_k=%d T=%d out of range", E, top_k, T);
    RouterParams p = {};
    p.wr = wr ? (const float*)wr->dev : nullptr;
    p.xn = xn;
    p.E = E;
    p.H = wr ? (int)wr->K : 0;
    p.T = T;
    p.top_k = top_k;
    p.scale = scale;
    p.mode = mode;
    p.ep_lo = ep_lo;
    p.ep_hi = ep_hi;
    p.logits = rt->logits;
    p.ids = rt->ids;
    p.weights = rt->weights;
    p.ticket = rt->ticket;
    p.n_active = rt->n_active;
    p.uexp = rt->uexp;
    p.uoff = rt->uoff;
    p.uassign = rt->uassign;
    p.sixteenths = sixteenths && T == 1;
    size_t smem = 0;
    if (norm) {
        if (!wr || T > 4) return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "router: rows to be normed need router weights, and are four at most");
        p.norm = *norm;
        smem = (size_t)T * p.H * 4;
        const int st = dc_kernel_setup(ctx, (const void*)k_router, 160 * 1024, "cudaFuncSetAttribute(k_router)");
        if (st != DC_B200_OK) return st;
    }
    return dc_launch(ctx, "k_router", k_router, dim3(wr ? (p.E + 1) / 2 : 1), dim3(256), smem, p);
}

// ------------------------------------------------------------ combine
// out[t][d] = sum over the token's assignments of w * down[assignment][d],
// added one at a time into a zeroed accumulator.  Order: routing order when
// T <= 4 and T*top_k <= 32 (cpu_backend_moe_ops.cpp:66,1247-1248,1578-1597),
// otherwise ascending expert id (moe_routing.cpp:647-676).  Assignments whose
// expert lives on another GPU are skipped (their share arrives by all-reduce).
// Whether a token's assignments are added up in routing order; else by ascending expert id.
__device__ __forceinline__ bool combine_as_routed(int T, int top_k) { return T <= 4 && T * top_k <= 32; }
// The order in which they are.
__device__ __forceinline__ void combine_order(const int32_t* ids, int T, int top_k, int t, int (&order)[MOE_MAX_K]) {
    for (int k = 0; k < top_k; ++k) order[k] = k;
    if (!combine_as_routed(T, top_k)) {
        for (int i = 1; i < top_k; ++i) {
            const int o = order[i], e = ids[t * top_k + o];
            int j = i - 1;
            while (j >= 0 && ids[t * top_k + order[j]] > e) {
                order[j + 1] = order[j];
                --j;
            }
            order[j + 1] = o;
        }
    }
}

__global__ void __launch_bounds__(256) k_moe_combine(const float* __restrict__ dn, const int32_t* __restrict__ ids,
                                                     const float* __restrict__ weights, int T, int top_k, int H,
                                                     int ep_lo, int ep_hi, float* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.y;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= H) return;
    int order[MOE_MAX_K];
    combine_order(ids, T, top_k, t, order);
    float sum = 0.0f;
    for (int k = 0; k < top_k; ++k) {
        const int a = t * top_k + order[k], e = ids[a];
        const float w = weights[a];
        if (e < ep_lo || e >= ep_hi || w == 0.0f) continue;
        sum = __fadd_rn(sum, __fmul_rn(w, dn[(size_t)a * H + d]));
    }
    out[(size_t)t * H + d] = sum;
}

int dc_launch_moe_combine(dc_ctx* ctx, const float* dn, const int32_t* ids, const float* weights, int T, int top_k,
                          int H, int ep_lo, int ep_hi, float* out) {
    return dc_launch(ctx, "k_moe_combine", k_moe_combine, dim3((H + 255) / 256, T), dim3(256), 0, dn, ids, weights, T,
                     top_k, H, ep_lo, ep_hi, out);
}

// One CTA per token: the combine above added to the residual, then RMSNorm and Q8_K blocks (k_rmsnorm_q8k's arithmetic).  A kernel of its
// own for the combine cost a launch of the step's chain and wrote and read the sum again.  Bound by that chain (its bytes are 82 KB a
// token): 4.4 us a layer at one token.
__global__ void __launch_bounds__(512) k_moe_combine_norm(const float* __restrict__ dn, const int32_t* __restrict__ ids, const float* __restrict__ weights,
                                                          int T, int top_k, int H, float* __restrict__ x, const float* __restrict__ nw, float eps,
                                                          float* __restrict__ xn_out, uint8_t* __restrict__ q8_out) {
    extern __shared__ __align__(16) float sx[];
    __shared__ double red[16];
    __shared__ float s_w[MOE_MAX_K];
    __shared__ int s_a[MOE_MAX_K];
    pdl_launch_dependents();
    const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n4 = H / 4;
    float4 w0 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < n4) w0 = reinterpret_cast<const float4*>(nw)[tid];
    pdl_wait();
    if (tid < top_k) {      // combine_order's places, all at once
        const int own = ids[t * top_k + tid];
        const float w = weights[t * top_k + tid];
        int at = tid;
        if (!combine_as_routed(T, top_k)) {
            at = 0;
            for (int k = 0; k < top_k; ++k) at += ids[t * top_k + k] < own;
        }
        s_a[at] = t * top_k + tid;
        s_w[at] = w;
    }
    __syncthreads();
    double ss = 0.0;
    for (int i = tid; i < n4; i += 512) {
        const float4 xv = reinterpret_cast<const float4*>(x + (size_t)t * H)[i];
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < top_k; k0 += 8) {
            float4 r[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)     // eight rows' loads in flight
                r[j] = reinterpret_cast<const float4*>(dn + (size_t)s_a[min(k0 + j, top_k - 1)] * H)[i];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (k0 + j >= top_k || s_w[k0 + j] == 0.0f) continue;
                const float w = s_w[k0 + j];
                s[0] = __fadd_rn(s[0], __fmul_rn(w, r[j].x));
                s[1] = __fadd_rn(s[1], __fmul_rn(w, r[j].y));
                s[2] = __fadd_rn(s[2], __fmul_rn(w, r[j].z));
                s[3] = __fadd_rn(s[3], __fmul_rn(w, r[j].w));
            }
        }
        const float4 v = make_float4(__fadd_rn(xv.x, s[0]), __fadd_rn(xv.y, s[1]), __fadd_rn(xv.z, s[2]), __fadd_rn(xv.w, s[3]));
        reinterpret_cast<float4*>(x + (size_t)t * H)[i] = v;
        reinterpret_cast<float4*>(sx)[i] = v;
        ss += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    double tot = 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) tot += red[i];
    const float mean = (float)(tot / (double)H);
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
    for (int i = tid; i < n4; i += 512) {
        const float4 v = reinterpret_cast<const float4*>(sx)[i], w = i == tid ? w0 : reinterpret_cast<const float4*>(nw)[i];
        const float4 y = make_float4(__fmul_rn(__fmul_rn(v.x, scale), w.x), __fmul_rn(__fmul_rn(v.y, scale), w.y),
                                     __fmul_rn(__fmul_rn(v.z, scale), w.z), __fmul_rn(__fmul_rn(v.w, scale), w.w));
        reinterpret_cast<float4*>(sx)[i] = y;
        if (xn_out) reinterpret_cast<float4*>(xn_out + (size_t)t * H)[i] = y;
    }
    if (!q8_out) return;
    __syncthreads();
    const int nb = H / DC_QK_K;
    for (int b = warp; b < nb; b += 16) quantize_block_q8k_warp<true>(sx + b * DC_QK_K, q8_out + ((size_t)t * nb + b) * DC_Q8F_BYTES, lane);
}

int dc_launch_moe_combine_norm(dc_ctx* ctx, const float* dn, const int32_t* ids, const float* weights, int T, int top_k, int H, float* x,
                               const float* norm_w, float eps, float* xn_out, uint8_t* q8_out) {
    return dc_launch(ctx, "k_moe_combine_norm", k_moe_combine_norm, dim3(T), dim3(512), (size_t)H * 4, dn, ids, weights, T, top_k, H, x, norm_w, eps, xn_out, q8_out);
}
