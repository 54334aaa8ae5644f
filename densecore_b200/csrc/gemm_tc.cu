// Batched MUL_MAT for prompt chunks (M >= 32 token rows): K-quant weights x Q8_K activations on the
// 5th-generation tensor cores, with block sums that are exact integers, so that the float steps per 256-value
// block are the CPU kernels' own
// (core/src/llm/matmul/batched_exec.cpp:1040-1240 serves these shapes on the CPU; per block
// sumf += (d*yd)*float(I); sumf -= (dmin*yd)*float(M), core/src/kernels/hwy/hwy_moe_quant.cc:248-253).
//
// The products are tcgen05.mma kind::f16 on whole numbers: a code times its sub-block's scale is one that fp16 holds exactly, so are the
// activation codes, and a sum of products that stays below 2^24 is exact in the f32 accumulator.  So the read-out gets floats:
//   Q4_K: q4 * sc (<= 945); the two halves of a block have an accumulator each (|sum| <= 945 * 127 * 128 < 2^24), whose sum rounds once: float(I).
//         The minimum term M = sum m_j * (sum of the token's codes in sub-block j) is one more product, of length 16: the minima (each twice) times the
//         sums of the token's codes over 16 values (<= 2048, exact), |M| <= 63 * 127 * 256.
//   Q6_K: q6 - 32 = (ql - 8) + 8 (2 qh - 3): sc (ql - 8) (<= 1024) with an accumulator for each half (<= 1024 * 128 * 128 = 2^24), and
//         8 sc (2 qh - 3) with one for the block, whose sums are multiples of 8 and stay below 2^27.  float(I) = the sum of the three, rounded once: where the
//         halves' sum reaches 2^24, a warp adds the three as integers.
// The weight operand lies in tensor memory (lane = row, 32 columns a quarter block, four slots), where its expander threads store it; only the
// activations take the way through shared memory, whose 128 bytes a cycle an operand of 128 rows from there would fill alone.
//
// One CTA per SM walks work items of 128 weight rows x two 64-token tiles over the whole reduction length, see k_gemm_tc below.
// The token side is prepared once per activation matrix by k_quantize_q8k_tiled (layout: dc_gemm_tc.h), so that every piece is a contiguous
// bulk copy.  No multicast load anywhere.
//
// Q4_K results are bit-equal to the GEMV path and the CPU oracle.  Q6_K adds one float term per block
// instead of the CPU small-batch kernel's eight lane partials (q6_small_batch.h:62-103): equal integers,
// a different float order, relative difference ~1e-7.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "dc_common.cuh"
#include "dc_gemm_tc.h"
#include "dc_internal.h"
#include "dc_launch.cuh"
#include "dc_tcgen05.cuh"

#define DC_TRY(expr)                       \
    do {                                   \
        int st_ = (expr);                  \
        if (st_ != DC_B200_OK) return st_; \
    } while (0)

namespace dc {

constexpr int TC_ROWS = 128;

struct GemmTcSeg {
    const uint8_t* w;      // rows of the matrix (expert 0)
    int N;                 // its rows
    int out_off;           // column offset of its outputs in a row of out
};

struct GemmTcParams {
    GemmTcSeg seg[3];      // matrices of one shape family (same K, row bytes, type) run in one launch: Q | K | V, gate | up
    int nseg;
    int row_bytes, K;
    const uint8_t* act;    // [K / 256][n_tt][TC_ACT_TILE]
    int n_tt;
    int n_slots;           // token slots that hold data (stores beyond are skipped)
    float* out;            // out[slot * ldo + row]
    int ldo;
    const int* tile_expert;   // optional [n_tt]: weights of tile t start at w + tile_expert[t] * estride; < 0: tile unused
    size_t estride;
    const int* slot_row;      // optional [n_tt * 64]: output row of every slot instead of the slot itself; < 0: none
    const int* pair_tile0;    // optional [grid.x]: first tile of the CTA's pair of neighbouring tiles (< 0: none) ...
    const int* pair_nset;     // ... and how many tiles of the pair exist (1 or 2); without it CTA i owns tiles 2i, 2i + 1
    int accumulate;           // out += result (one float add) instead of out = result
    float one;                // 1, which the compiler must not know (see fma2_rn)
    int tiles_x, tiles_y;     // work items: token-tile pairs x row tiles (of all matrices of the launch)
    int* err;
};

// Packed single precision (two lanes per instruction), each lane rounded to nearest like the scalar instruction.  An addition behind a
// multiplication is written as fma2_rn(product, one, sum) with a `one` from the kernel's parameters: a packed add there was seen to round
// once, as if fused with the multiplication.
__device__ __forceinline__ float2 mul2_rn(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n mul.rn.f32x2 rd, ra, rb;\n mov.b64 {%0, %1}, rd;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 add2_rn(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n add.rn.f32x2 rd, ra, rb;\n mov.b64 {%0, %1}, rd;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 fma2_rn(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n .reg .b64 ra, rb, rc, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n mov.b64 rc, {%6, %7};\n"
        " fma.rn.f32x2 rd, ra, rb, rc;\n mov.b64 {%0, %1}, rd;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// ---- activation side ---------------------------------------------------------------------------------
// One warp per (token slot, 256-value block): Q8_K codes (bit-equal to the row quantiser) into the tile
// layout of dc_gemm_tc.h, block scale into the tile's tail.  slot_token (optional) maps a slot to its source
// row, < 0 or beyond n_rows: the slot is left as it is.  (What an unused slot holds stays in its own column of the products: gate and up store it into the
// slot's own row, which nobody reads, the down product stores nothing of it.  A third of a prompt's expert slots are such; with zeros written there the three
// launches of a layer took 80 us for 2011 tokens, now 73.)
__global__ void __launch_bounds__(256) k_quantize_q8k_tiled(const float* __restrict__ x, int ldx, int n_rows, int K,
                                                            uint8_t* __restrict__ act, int n_tt,
                                                            const int* __restrict__ slot_token) {
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = K / DC_QK_K;
    const long long total = (long long)n_tt * TC_NTOK * nb;
    for (long long item = (long long)blockIdx.x * 8 + warp; item < total; item += (long long)gridDim.x * 8) {
        const int b = (int)(item % nb);
        const int slot = (int)(item / nb);
        int row = slot_token ? slot_token[slot] : slot;
        if (row >= n_rows) row = -1;
        if (row < 0) continue;
        uint8_t* tile = act + ((size_t)b * n_tt + slot / TC_NTOK) * TC_ACT_TILE;
        uint32_t w0, w1, bw;
        float d;
        const float4* src = reinterpret_cast<const float4*>(x + (size_t)row * ldx + (size_t)b * DC_QK_K + 8 * lane);
        const float4 a = src[0], c = src[1];
        const float v[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
        q8k_block_core(v, lane, w0, w1, bw, d);
        tc_act_store(tile, slot % TC_NTOK, lane, w0, w1, bw, d);
    }
}

// ---- the kernel -----------------------------------------------------------------------------------------
// The three jobs of a block (expanding the weight operand, issuing products, reading the accumulators out) run on different warps of one CTA per
// SM and overlap.  A work item is 128 rows x two 64-token tiles; the CTA walks its items round robin, and every ring slot and barrier phase is
// picked by the number of the block, which runs on across items, so an item's first blocks are expanded while the item before is read out.
//   warps 0-7    expanders: thread r of four warps turns its row's quarter block into the 32 columns of an operand slot.  Q4_K: either four take
//                every second quarter, expanded in registers before the slot is free; Q6_K: the lower four bits, the upper two
//   warps 8-23   read-out: warp w owns TMEM lane quarter w % 4 and sixteen tokens of either tile
//   warps 24, 25 issue the products
//   warp 26      loads the token tiles (three blocks ahead)
// Tensor memory: two sets of three 64-column accumulators, one per token tile (a lone tile takes them in turn), so that one is read out while the
// other's products run, and the four operand slots.
// What bounds it: the chain of a block (operand slot free, stored, multiplied, read out, accumulators free), each hand-over 150 to 400 cycles, while every SM
// sub-partition is about half busy (packed multiply-adds of the read-out, expansion); without the read-out's work a block takes 10 % less, without the
// expansion's 16 %, without either 28 %.  Measured, us, against the int8 form of this kernel (operands in shared memory, 13 instead of 4 instructions per element
// and block in the read-out): Q4_K 4096 x 2048 by 1531 tokens 70 -> 47, Q6_K 114 -> 92; 2048 x 4096 by 300 tokens 45 -> 29 and 82 -> 62, 2048 x 768 by 64 11 -> 8 and 18 -> 13.  Tried:
// accumulators of 128 tokens (one set only, 63 us); eight read-out warps, or four expanders (61); one issuing warp (48); operand slots of half a block (60).
constexpr int TC_EXPANDERS = 8, TC_READERS = 16;
constexpr int TC_WARP_MMA = TC_EXPANDERS + TC_READERS;
constexpr int TC_THREADS = (TC_WARP_MMA + 4) * 32;         // (the last warp only gives its registers)
// Registers a thread at launch, of the read-out and of the last four warps once they have shared theirs out anew; expanders keep the launch's.  What the read-out takes has
// to be what the others give: from a launch with fewer registers it would wait for more without end, so the launcher refuses any other build.
constexpr int TC_LAUNCH_REGS = 72, TC_READ_REGS = 80, TC_REST_REGS = 40;
static_assert(TC_EXPANDERS * TC_LAUNCH_REGS + TC_READERS * TC_READ_REGS + 4 * TC_REST_REGS <= (TC_THREADS / 32) * TC_LAUNCH_REGS, "the launch's registers");
static_assert(TC_EXPANDERS % 4 == 0 && TC_READERS % 4 == 0, "whole warpgroups");
constexpr int TC_B_STAGES = 3;
constexpr uint32_t TC_SET = 3 * TC_NTOK;                   // columns of a set of accumulators
constexpr uint32_t TC_COL_A = 2 * TC_SET;                  // first operand column

// mbarriers of the kernel, as indexes from the first one
enum TcBar { A_FULL = 0, A_FREE = 4, B_FULL = 8, B_FREE = 11, S_FULL = 14, D_FULL = 22, ACC_FULL = 26, ACC_FREE = 28, DRAIN = 30, TC_NBARS = 32 };

constexpr uint32_t TC_TILE = TC_B_Q + 2 * TC_SUM_HALF;                     // a token tile without its scales
constexpr uint32_t TC_SB = 0;                                              // [3][two tiles]
constexpr uint32_t TC_SM = TC_SB + TC_B_STAGES * 2 * TC_TILE;              // the rows' minima as an operand: [half][row][16 bytes]
constexpr uint32_t TC_SSC = TC_SM + 4096;                                  // [8][two tiles] block scales
constexpr uint32_t TC_SD = TC_SSC + 8 * 2 * TC_ACT_SCALES;                 // [4][128] d, -dmin of the rows
constexpr uint32_t TC_SBAR = TC_SD + 4 * 128 * 8;
constexpr size_t TC_SMEM = TC_SBAR + TC_NBARS * 8 + 16 + 1024;             // the swizzled tiles start on a 1024-byte boundary

struct TcTile {       // one work item: 128 rows of one matrix x a pair of neighbouring 64-token tiles of one expert
    bool live;
    int tt0, nset, seg, N, row0;
    const uint8_t* wbase;
};
__device__ __forceinline__ TcTile tc_tile_at(const GemmTcParams& p, int t) {
    TcTile ti;
    ti.live = false;
    const int px = t % p.tiles_x, py = t / p.tiles_x;
    if (p.pair_tile0) {
        ti.tt0 = p.pair_tile0[px];
        if (ti.tt0 < 0) return ti;
        ti.nset = p.pair_nset[px];
    } else {
        ti.tt0 = 2 * px;
        ti.nset = min(2, p.n_tt - ti.tt0);
    }
    const int expert = p.tile_expert ? p.tile_expert[ti.tt0] : 0;
    if (expert < 0) return ti;
    int seg = 0, rt = py;
    while (seg + 1 < p.nseg && rt >= (p.seg[seg].N + TC_ROWS - 1) / TC_ROWS) {
        rt -= (p.seg[seg].N + TC_ROWS - 1) / TC_ROWS;
        ++seg;
    }
    ti.seg = seg;
    ti.N = p.seg[seg].N;
    ti.row0 = rt * TC_ROWS;
    ti.wbase = p.seg[seg].w + (size_t)expert * p.estride;
    ti.live = true;
    return ti;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
__device__ __forceinline__ __half2 h2_of(float x) { return __float2half2_rn(x); }

// 4 x 8 nibbles of a Q4_K row -> 16 operand columns.  0x6400 + n are the bits of 1024 + n, and (1024 + n) * s - 1024 * s is n * s exactly in one
// fused multiply-add (s <= 63; high nibbles stay in place: (1024 + 16 n) * (s / 16) - 64 s).
struct Q4Scale {
    __half2 s, n, s16, n16;      // of the low nibbles' sub-block: s, -1024 s; of the high nibbles': s / 16, -64 s
    __device__ __forceinline__ void set(uint32_t scw) {      // the scales in the lower two bytes
        const __half2 k = h2_of(-1024.0f);
        const __half2 lo = __hadd2(bits_h2(__byte_perm(scw, 0x64u, 0x4040)), k), hi = __hadd2(bits_h2(__byte_perm(scw, 0x64u, 0x4141)), k);
        s = lo;
        n = __hmul2(lo, k);
        s16 = __hmul2(hi, h2_of(0.0625f));
        n16 = __hmul2(hi, h2_of(-64.0f));
    }
};
__device__ __forceinline__ void q4_columns(uint4 q, const Q4Scale& c, uint32_t (&v)[16]) {
    const uint32_t in[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t w = in[k], w8 = w >> 8;
        v[4 * k] = h2_bits(__hfma2(bits_h2((w & 0x000F000Fu) | 0x64006400u), c.s, c.n));
        v[4 * k + 1] = h2_bits(__hfma2(bits_h2((w8 & 0x000F000Fu) | 0x64006400u), c.s, c.n));
        v[4 * k + 2] = h2_bits(__hfma2(bits_h2((w & 0x00F000F0u) | 0x64006400u), c.s16, c.n16));
        v[4 * k + 3] = h2_bits(__hfma2(bits_h2((w8 & 0x00F000F0u) | 0x64006400u), c.s16, c.n16));
    }
}
// Eight words of either 32-value run of a quarter (`second`: the later quarter of a half block), four at a time: w the words of the first run,
// x of the second, with 16-value scales s0 and s1 -> 16 columns of sc (ql - 8); nibbles stay in place.
__device__ __forceinline__ void q6_low_columns(const uint32_t* w, const uint32_t* x, float s0, float s1, bool second, uint32_t (&v)[16]) {
    const __half2 f0 = h2_of(second ? s0 * 0.0625f : s0), f1 = h2_of(second ? s1 * 0.0625f : s1), k = h2_of(second ? -1152.0f : -1032.0f);
    const uint32_t m = second ? 0x00F000F0u : 0x000F000Fu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[4 * i] = h2_bits(__hmul2(__hadd2(bits_h2((w[i] & m) | 0x64006400u), k), f0));
        v[4 * i + 1] = h2_bits(__hmul2(__hadd2(bits_h2(((w[i] >> 8) & m) | 0x64006400u), k), f0));
        v[4 * i + 2] = h2_bits(__hmul2(__hadd2(bits_h2((x[i] & m) | 0x64006400u), k), f1));
        v[4 * i + 3] = h2_bits(__hmul2(__hadd2(bits_h2(((x[i] >> 8) & m) | 0x64006400u), k), f1));
    }
}
// The same of 8 sc (2 qh - 3).  The two bits of quadrant i of a half block lie at bits 2 i of a byte: u (2 qh - 3) with u = 1 << (2 i - 1) (quadrant 0
// moved up a bit) after the bias 1024 + 3 u, then times 8 sc / u.
__device__ __forceinline__ void q6_high_columns(const uint32_t* w, float s0, float s1, bool second, uint32_t (&v)[16]) {
    const __half2 k0 = h2_of(second ? -1048.0f : -1027.0f), k1 = h2_of(second ? -1120.0f : -1030.0f);
    const __half2 f0 = h2_of(second ? s0 : 8.0f * s0), f1 = h2_of(second ? 0.25f * s1 : 4.0f * s1);
    const uint32_t m0 = second ? 0x00300030u : 0x00060006u, m1 = second ? 0x00C000C0u : 0x000C000Cu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t a = second ? w[i] : w[i] << 1, a8 = second ? w[i] >> 8 : w[i] >> 7;
        v[4 * i] = h2_bits(__hmul2(__hadd2(bits_h2((a & m0) | 0x64006400u), k0), f0));
        v[4 * i + 1] = h2_bits(__hmul2(__hadd2(bits_h2((a8 & m0) | 0x64006400u), k0), f0));
        v[4 * i + 2] = h2_bits(__hmul2(__hadd2(bits_h2((w[i] & m1) | 0x64006400u), k1), f1));
        v[4 * i + 3] = h2_bits(__hmul2(__hadd2(bits_h2(((w[i] >> 8) & m1) | 0x64006400u), k1), f1));
    }
}

template <int TYPE>
__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_tc(const GemmTcParams p) {
    constexpr bool Q4 = TYPE == DC_TYPE_Q4_K;
    constexpr int BB = Q4 ? DC_Q4K_BYTES : DC_Q6K_BYTES;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ uint32_t s_tmem;
    const uint32_t sm = (smem_u32(smem_raw) + 1023u) & ~1023u;
    auto bar = [sm](int which, int i = 0) -> uint32_t { return sm + TC_SBAR + 8u * (uint32_t)(which + i); };
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nb = p.K / DC_QK_K, total = p.tiles_x * p.tiles_y;

    if (warp == TC_WARP_MMA) {
        tmem_alloc(smem_u32(&s_tmem), 512);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < TC_NBARS; ++i) mbar_init(bar(i), i < A_FREE || (i >= D_FULL && i < ACC_FULL) ? 4 : i >= ACC_FREE && i < DRAIN ? TC_READERS : (i >= B_FREE && i < S_FULL) || (i >= ACC_FULL && i < ACC_FREE) ? 2 : 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_wait();      // (the set-up above overlaps the quantiser's end)
    auto wait = [](uint32_t b, uint32_t parity) { return mbar_wait_warp(b, parity); };
    // Every role walks the same list of items (this CTA's share, round robin) and counts blocks across them (g).  Why no slot is overwritten too
    // early: products of block g run only when the read-out has released the last block of that set of accumulators, g - 1 or, in a lone tile, g - 2,
    // behind its last reads of that block's d, dmin and scales.  Row constants of block g are stored behind products of g - 1, so those
    // of g - 3 and before are free: a ring of four.  Scales of block g are loaded behind products of g - 3: those of g - 5 and before are free: a ring of eight.
    if (warp < TC_EXPANDERS) {
        // ------------------------------------------------------------------ expanders
        const int r = tid & 127, grp = warp >> 2;
        const uint32_t t_a = tmem + TC_COL_A + ((uint32_t)(32 * (warp & 3)) << 16);
        auto filled = [&](int slot) {
            __syncwarp();
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(A_FULL, slot));
        };
        int g = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x) {
            const TcTile ti = tc_tile_at(p, t);
            if (!ti.live) continue;
            const uint8_t* rp = ti.wbase + (size_t)min(ti.row0 + r, ti.N - 1) * p.row_bytes;
            if constexpr (Q4) {
                // this warp's quarters of a block: grp and grp + 2; a quarter's raw quants are requested one turn ahead
                const uint4* b = reinterpret_cast<const uint4*>(rp);
                const uint4* from = b + 1 + 2 * grp;
                uint4 H = __ldg(b), q0 = __ldg(from), q1 = __ldg(from + 1);
#pragma unroll 1
                for (int i = 0; i < 2 * nb; ++i) {
                    const int j = i & 1, slot = grp + 2 * j;
                    // the 6-bit scales of sub-blocks 4 j .. 4 j + 3, four to a word (get_scale_min_k4 of ggml's K-quants on packed bytes)
                    const uint32_t scw = j ? ((H.w & 0x0F0F0F0Fu) | (((H.y >> 6) & 0x03030303u) << 4)) : (H.y & 0x3F3F3F3Fu);
                    Q4Scale sc;
                    sc.set(scw >> (16 * grp));
                    uint32_t v[2][16];
                    q4_columns(q0, sc, v[0]);
                    q4_columns(q1, sc, v[1]);
                    const bool more = i + 1 < 2 * nb;
                    from += j ? 5 : 4;
                    if (more) {
                        q0 = __ldg(from);
                        q1 = __ldg(from + 1);
                    }
                    if (!wait(bar(A_FREE, slot), (g & 1) ^ 1)) goto gave_up;      // (the first passes)
                    tc_fence_after();
                    tmem_st16(t_a + 32 * slot, v[0]);
                    tmem_st16(t_a + 32 * slot + 16, v[1]);
                    if (!j && grp == 0) {
                        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(sm + TC_SD + ((g & 3) * 128 + r) * 8), "f"(fp16_bits_to_float((uint16_t)(H.x & 0xFFFF))),
                                     "f"(-fp16_bits_to_float((uint16_t)(H.x >> 16)))
                                     : "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(D_FULL, g & 3));
                    }
                    if (j) {
                        if (grp == 1) {
                            // minima of sub-blocks 0..3, 4..7 as pairs of equal fp16 numbers (the product that read the last ones is done, as the slot's is)
                            const uint32_t mw[2] = {H.z & 0x3F3F3F3Fu, ((H.w >> 4) & 0x0F0F0F0Fu) | (((H.z >> 6) & 0x03030303u) << 4)};
                            const __half2 k = h2_of(-1024.0f);
#pragma unroll
                            for (int n = 0; n < 2; ++n)
                                sts128(sm + TC_SM + n * 2048 + (r >> 3) * 128 + (r & 7) * 16, h2_bits(__hadd2(bits_h2(__byte_perm(mw[n], 0x64u, 0x4040)), k)),
                                       h2_bits(__hadd2(bits_h2(__byte_perm(mw[n], 0x64u, 0x4141)), k)), h2_bits(__hadd2(bits_h2(__byte_perm(mw[n], 0x64u, 0x4242)), k)),
                                       h2_bits(__hadd2(bits_h2(__byte_perm(mw[n], 0x64u, 0x4343)), k)));
                            fence_async_smem();
                        }
                        ++g;
                        b += 9;
                        if (more) H = __ldg(b);
                    }
                    filled(slot);
                }
            } else {
                // 210-byte blocks at 2-byte aligned addresses: aligned 32-bit loads and a funnel shift; a half block is requested ahead
                uint32_t raw[17], ws[3], wd = 0;      // 17 words of lower bits, or 9 of upper
                auto fetch = [&](int i) {      // half i & 1 of block i / 2
                    const uintptr_t a = (uintptr_t)(rp + (size_t)(i >> 1) * BB);
                    const int h = i & 1;
                    const uint32_t* bs = reinterpret_cast<const uint32_t*>((a + 192 + 8 * h) & ~(uintptr_t)3);
#pragma unroll
                    for (int k = 0; k < 3; ++k) ws[k] = __ldg(bs + k);
                    if (grp == 0) {
                        const uint32_t* bl = reinterpret_cast<const uint32_t*>((a + 64 * h) & ~(uintptr_t)3);
#pragma unroll
                        for (int k = 0; k < 17; ++k) raw[k] = __ldg(bl + k);
                        wd = __ldg(reinterpret_cast<const uint32_t*>((a + 208) & ~(uintptr_t)3));
                    } else {
                        const uint32_t* bh = reinterpret_cast<const uint32_t*>((a + 128 + 32 * h) & ~(uintptr_t)3);
#pragma unroll
                        for (int k = 0; k < 9; ++k) raw[k] = __ldg(bh + k);
                    }
                };
                fetch(0);
#pragma unroll 1
                for (int i = 0; i < 2 * nb; ++i) {
                    const int h = i & 1;
                    const uint32_t sh = (uint32_t)((uintptr_t)(rp + (size_t)(i >> 1) * BB) & 2u) * 8u;       // every field of the block shares the 2-byte phase
                    uint32_t w[16], scw[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) scw[k] = __funnelshift_r(ws[k], ws[k + 1], sh);
                    if (grp == 0) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) w[k] = __funnelshift_r(raw[k], raw[k + 1], sh);
                        if (h == 0) {
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(sm + TC_SD + ((g & 3) * 128 + r) * 8), "f"(fp16_bits_to_float((uint16_t)((wd >> sh) & 0xFFFFu))) : "memory");
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar(D_FULL, g & 3));
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) w[k] = __funnelshift_r(raw[k], raw[k + 1], sh);
                    }
                    if (i + 1 < 2 * nb) fetch(i + 1);
#pragma unroll
                    for (int gl = 0; gl < 2; ++gl) {      // quarter 2 h + gl: quadrants 2 gl and 2 gl + 1 of the half
                        const int slot = 2 * gl + grp;      // filled twice a block
                        if (!wait(bar(A_FREE, slot), h ^ 1)) goto gave_up;      // (the first passes)
                        tc_fence_after();
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {      // words 0..3, 4..7: one 16-value group of either quadrant
                            const float s0 = (float)(int8_t)(scw[gl] >> (8 * hf)), s1 = (float)(int8_t)(scw[gl] >> (16 + 8 * hf));
                            uint32_t v[16];
                            if (grp == 0) q6_low_columns(w + 4 * hf, w + 8 + 4 * hf, s0, s1, gl, v);
                            else q6_high_columns(w + 4 * hf, s0, s1, gl, v);
                            tmem_st16(t_a + 32 * slot + 16 * hf, v);
                        }
                        filled(slot);
                    }
                    g += h;
                }
            }
        }
    } else if (warp < TC_WARP_MMA) {
        // ------------------------------------------------------------------ read-out
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TC_READ_REGS));
        // every warp reads sixteen tokens of either tile: a set of accumulators is free again sooner than with eight warps for each tile
        const int tok0 = 16 * ((warp - TC_EXPANDERS) >> 2);
        const uint32_t t_lane = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + tok0;
        const float2 one = make_float2(p.one, p.one);
        int g = 0;
        uint32_t phase = 0;      // bit i: of set i's next use
        for (int t = blockIdx.x; t < total; t += gridDim.x) {
            bool two;
            {
                const TcTile ti = tc_tile_at(p, t);
                if (!ti.live) continue;
                two = ti.nset == 2;
            }
            float2 sum[2][8];
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[i >> 3][i & 7] = make_float2(0.0f, 0.0f);
#pragma unroll 1
            for (int kb = 0; kb < nb; ++kb, ++g) {
                float2 d2, dm2;
#pragma unroll
                for (int th = 0; th < 2; ++th) {
                    if (th && !two) break;
                    const int set = th ? 1 : two ? 0 : kb & 1;
                    // some lanes wait for the accumulators, some for d and dmin, some for the scales
                    const uint32_t b = th || lane & 1 ? bar(ACC_FULL, set) : lane & 2 ? bar(D_FULL, g & 3) : bar(S_FULL, g & 7);
                    if (!wait(b, th || lane & 1 ? (phase >> set) & 1 : lane & 2 ? (g >> 2) & 1 : (g >> 3) & 1)) goto gave_up;
                    phase ^= 1u << set;
                    tc_fence_after();
                    const uint32_t yds = sm + TC_SSC + ((g & 7) * 2 + th) * TC_ACT_SCALES + 4 * tok0, col = t_lane + set * TC_SET;
                    // eight tokens at a time; the next loads are on their way while the float terms of the last are made
                    int x0[8], x1[8];
                    tmem_ld8(col, x0);
                    tmem_ld8(col + TC_NTOK, x1);
                    if (th == 0) {
                        const uint2 dd = lds64(sm + TC_SD + ((g & 3) * 128 + 32 * (warp & 3) + lane) * 8);
                        d2 = make_float2(__uint_as_float(dd.x), __uint_as_float(dd.x));
                        dm2 = make_float2(__uint_as_float(dd.y), __uint_as_float(dd.y));
                    }
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        int x2[8];
                        float2 yd[4];
                        auto scales = [&]() {
                            const uint4 ya = lds128(yds + 32 * c), yb = lds128(yds + 32 * c + 16);
                            yd[0] = make_float2(__uint_as_float(ya.x), __uint_as_float(ya.y)), yd[1] = make_float2(__uint_as_float(ya.z), __uint_as_float(ya.w));
                            yd[2] = make_float2(__uint_as_float(yb.x), __uint_as_float(yb.y)), yd[3] = make_float2(__uint_as_float(yb.z), __uint_as_float(yb.w));
                        };
                        if (Q4) scales();
                        auto pair = [](const int (&v)[8], int i) { return make_float2(__int_as_float(v[2 * i]), __int_as_float(v[2 * i + 1])); };
                        tmem_ld_wait(x0);
                        tmem_loaded(x1);
                        tmem_ld8(col + 2 * TC_NTOK + 8 * c, x2);
                        float2 x[4];
                        float most = 0.0f;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float2& s = sum[th][4 * c + i];
                            x[i] = add2_rn(pair(x0, i), pair(x1, i));
                            if (!Q4) most = fmaxf(most, fmaxf(fabsf(x[i].x), fabsf(x[i].y)));
                            if (Q4) s = fma2_rn(mul2_rn(mul2_rn(d2, yd[i]), x[i]), one, s);
                        }
                        tmem_ld_wait(x2);
                        if constexpr (!Q4) {
                            if (__any_sync(0xffffffffu, most >= 16777216.0f)) {      // a sum of the halves may have been rounded: all three anew, as integers
                                int I[8];
#pragma unroll
                                for (int i = 0; i < 8; ++i) I[i] = __float2int_rn(__int_as_float(x2[i]));
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    tmem_ld8(col + h * TC_NTOK + 8 * c, x0);
                                    tmem_ld_wait(x0);
#pragma unroll
                                    for (int i = 0; i < 8; ++i) I[i] += __float2int_rn(__int_as_float(x0[i]));
                                }
#pragma unroll
                                for (int i = 0; i < 4; ++i) x[i] = make_float2(__int2float_rn(I[2 * i]), __int2float_rn(I[2 * i + 1]));
                            } else {
#pragma unroll
                                for (int i = 0; i < 4; ++i) x[i] = add2_rn(x[i], pair(x2, i));
                            }
                            scales();
                        }
                        if (c == 0) {
                            tmem_ld8(col + 8, x0);
                            tmem_ld8(col + TC_NTOK + 8, x1);
                        } else {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar(ACC_FREE, set));
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float2& s = sum[th][4 * c + i];
                            if (Q4) s = fma2_rn(mul2_rn(mul2_rn(dm2, yd[i]), pair(x2, i)), one, s);
                            else s = fma2_rn(mul2_rn(mul2_rn(d2, yd[i]), x[i]), one, s);
                        }
                    }
                }
            }
            int again = t;      // (the item looked up anew: its values would hold registers through the loop)
            asm volatile("" : "+r"(again));
            const TcTile ti = tc_tile_at(p, again);
            const int row = ti.row0 + 32 * (warp & 3) + lane;
            const uint64_t out = reinterpret_cast<uint64_t>(p.out + p.seg[ti.seg].out_off + row);
            const uint32_t pitch = 4u * (uint32_t)p.ldo;
            // output rows of the sixteen slots of either tile, one to a lane (little code: what the blocks' loops need stays in the instruction caches)
            const int slot = ti.tt0 * TC_NTOK + (lane & 16 ? TC_NTOK : 0) + tok0 + (lane & 15);
            const int at = slot < p.n_slots && (two || lane < 16) ? (p.slot_row ? p.slot_row[slot] : slot) : -1;
            const bool live = row < ti.N;
#pragma unroll
            for (int th = 0; th < 2; ++th) {
                if (th && !two) break;
                float old[16];
                if (p.accumulate) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int to = __shfl_sync(0xffffffffu, at, 16 * th + i);
                        if (live && to >= 0) old[i] = *reinterpret_cast<const float*>(out + (uint64_t)(uint32_t)to * pitch);
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float& x = i & 1 ? sum[th][i >> 1].y : sum[th][i >> 1].x;
                        x = __fadd_rn(old[i], x);
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int to = __shfl_sync(0xffffffffu, at, 16 * th + i);
                    if (live && to >= 0) *reinterpret_cast<float*>(out + (uint64_t)(uint32_t)to * pitch) = i & 1 ? sum[th][i >> 1].y : sum[th][i >> 1].x;
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REST_REGS));
        const bool one = elect_one();
        if (warp < TC_WARP_MMA + 2) {
            // ------------------------------------------------------------------ products
            // Two warps: Q4_K: the halves of a block; Q6_K: the lower and the upper bits.  Either has accumulators of its own, so they need no order.  (A wait takes 100
            // cycles and more even where nothing is to wait for, and a warp has six a block.)
            const int h = warp - TC_WARP_MMA;
            int st = 0;
            uint32_t st_phase = 0, a_phase = 0, phase = 3;      // of the stage, of the operand slots, bit i: of set i's last use (the first passes)
            bool ok = true;
            constexpr uint32_t idesc = umma_idesc_f16(TC_ROWS, TC_NTOK);
            auto set_free = [&](int set) {
                const bool is = wait(bar(ACC_FREE, set), (phase >> set) & 1);
                phase ^= 1u << set;
                return is;
            };
            // a quarter block of a tile (its descriptor) from an operand slot into the accumulator at d
            auto part = [&](uint32_t d, uint64_t tile, int slot, bool first) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_f16_ts(d, tmem + TC_COL_A + 32 * slot + 8 * k, tile + 2 * k, idesc, !first || k > 0);
            };
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                const TcTile ti = tc_tile_at(p, t);
                if (!ti.live) continue;
                const bool two = ti.nset == 2;
#pragma unroll 1
                for (int kb = 0; kb < nb && ok; ++kb) {
                    const int set = two ? 0 : kb & 1;      // of the first tile
                    const uint32_t at = sm + TC_SB + st * (2 * TC_TILE), d0 = tmem + set * TC_SET, d1 = tmem + TC_SET;
                    const uint64_t tiles = umma_desc_sw128(at, 1024);
                    ok = wait(bar(B_FULL, st), st_phase) && set_free(set);
                    if constexpr (Q4) {
                        const uint64_t mine = tiles + h * (2 * TC_QUARTER / 16), sums = umma_desc_plain(at + TC_B_Q, TC_SUM_HALF, 128), m = umma_desc_plain(sm + TC_SM, 2048, 128);
                        const uint32_t to = h * TC_NTOK;
#pragma unroll
                        for (int th = 0; th < 2; ++th) {
                            if (th && !two) break;
                            if (th) ok = ok && set_free(1);
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                if (th == 0) ok = ok && wait(bar(A_FULL, 2 * h + j), a_phase);
                                if (!ok) break;
                                tc_fence_after();
                                if (one) {
                                    const uint32_t d = th ? d1 : d0;
                                    part(d + to, mine + (th * TC_TILE + j * TC_QUARTER) / 16, 2 * h + j, j == 0);
                                    if (j == 1) {
                                        if (h == 1) umma_f16(d + 2 * TC_NTOK, m, sums + th * TC_TILE / 16, idesc, 0);
                                        umma_commit(bar(ACC_FULL, th ? 1 : set));
                                    }
                                    if (th || !two) umma_commit(bar(A_FREE, 2 * h + j));
                                }
                            }
                        }
                    } else {
                        // an operand slot serves both tiles before it is filled anew
                        if (two) ok = ok && set_free(1);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int slot = 2 * (q & 1) + h;
                            ok = ok && wait(bar(A_FULL, slot), q >> 1);
                            if (!ok) break;
                            tc_fence_after();
                            if (one) {
                                const uint32_t to = (h ? 2 : q >> 1) * TC_NTOK;
                                const bool first = q == 0 || (h == 0 && q == 2);
                                part(d0 + to, tiles + q * (TC_QUARTER / 16), slot, first);
                                if (q == 3) umma_commit(bar(ACC_FULL, set));
                                if (two) {
                                    part(d1 + to, tiles + (TC_TILE + q * TC_QUARTER) / 16, slot, first);
                                    if (q == 3) umma_commit(bar(ACC_FULL, 1));
                                }
                                umma_commit(bar(A_FREE, slot));
                            }
                        }
                    }
                    if (ok && one) umma_commit(bar(B_FREE, st));
                    a_phase ^= 1;
                    if (++st == TC_B_STAGES) {
                        st = 0;
                        st_phase ^= 1;
                    }
                }
            }
            if (!ok) {      // products in flight still read shared and tensor memory
                if (one) umma_commit(bar(DRAIN, h));
                mbar_wait(bar(DRAIN, h), 0, nullptr);
                goto gave_up;
            }
        } else if (warp == TC_WARP_MMA + 2) {
            // ------------------------------------------------------------------ token tiles
            int g = 0, st = 0;
            uint32_t st_phase = 1;      // of the stage's last use (the first passes)
            for (int t = blockIdx.x; t < total; t += gridDim.x) {
                const TcTile ti = tc_tile_at(p, t);
                if (!ti.live) continue;
                for (int kb = 0; kb < nb; ++kb, ++g) {
                    if (!wait(bar(B_FREE, st), st_phase)) {
                        // copies of the last blocks may still be on their way
                        for (int o = max(0, g - TC_B_STAGES); o < g; ++o) mbar_wait(bar(B_FULL, o % TC_B_STAGES), (o / TC_B_STAGES) & 1, nullptr);
                        for (int o = max(0, g - 8); o < g; ++o) mbar_wait(bar(S_FULL, o & 7), (o >> 3) & 1, nullptr);
                        goto gave_up;
                    }
                    if (one) {
                        const uint8_t* src = p.act + ((size_t)kb * p.n_tt + ti.tt0) * TC_ACT_TILE;
                        const uint32_t dst = sm + TC_SB + st * (2 * TC_TILE), dss = sm + TC_SSC + (g & 7) * (2 * TC_ACT_SCALES);
                        constexpr uint32_t n = Q4 ? TC_TILE : TC_B_Q;
                        mbar_expect_tx(bar(B_FULL, st), ti.nset * n);
                        mbar_expect_tx(bar(S_FULL, g & 7), ti.nset * TC_ACT_SCALES);
                        bulk_g2s(dst, src, n, bar(B_FULL, st));
                        bulk_g2s(dss, src + TC_TILE, TC_ACT_SCALES, bar(S_FULL, g & 7));
                        if (ti.nset == 2) {
                            bulk_g2s(dst + TC_TILE, src + TC_ACT_TILE, n, bar(B_FULL, st));
                            bulk_g2s(dss + TC_ACT_SCALES, src + TC_ACT_TILE + TC_TILE, TC_ACT_SCALES, bar(S_FULL, g & 7));
                        }
                    }
                    if (++st == TC_B_STAGES) {
                        st = 0;
                        st_phase ^= 1;
                    }
                }
            }
        }
    }
    if (false) {
    gave_up:
        if (p.err) atomicExch(p.err, DC_ERR_MBAR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TC_WARP_MMA) tmem_dealloc(tmem, 512);
}

}  // namespace dc

using namespace dc;

size_t dc_gemm_tc_act_bytes(int n_slots, int K) {
    const int n_tt = (n_slots + TC_NTOK - 1) / TC_NTOK;
    return (size_t)(K / DC_QK_K) * n_tt * TC_ACT_TILE;
}

int dc_gemm_tc_tiles(int n_slots) { return (n_slots + TC_NTOK - 1) / TC_NTOK; }

// x [n_rows, K] f32 (row stride ldx) -> tiled Q8_K activations for n_tt token tiles; slot_token: optional
// device array [n_tt * 64] mapping slots to rows of x.
int dc_launch_quantize_q8k_tiled(dc_ctx* ctx, const float* x, int ldx, int n_rows, int K, uint8_t* act, int n_tt,
                                 const int* slot_token) {
    if (K % DC_QK_K || ldx % 4 || ((uintptr_t)x & 15)) return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "quantize_q8k_tiled: K=%d ldx=%d", K, ldx);
    const long long items = (long long)n_tt * TC_NTOK * (K / DC_QK_K);
    long long blocks = (items + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_quantize_q8k_tiled<<<(unsigned)blocks, 256, 0, ctx->stream>>>(x, ldx, n_rows, K, act, n_tt, slot_token);
    return dc_check_cuda(ctx, cudaGetLastError(), "k_quantize_q8k_tiled");
}

bool dc_gemm_tc_supports(const dc_weight* w) {
    if (w->type == DC_TYPE_Q4_K) return ((uintptr_t)w->dev & 15) == 0 && w->row_bytes % 16 == 0;
    return w->type == DC_TYPE_Q6_K && ((uintptr_t)w->dev & 1) == 0;
}

// out[slot * ldo + row] = sum over K of w[row] . act[slot] for rows [0, N) and slots [0, n_slots); with tile_expert,
// token tile t uses the matrix of expert tile_expert[t] (skipped when negative).
// Up to three matrices of one shape family (same type, K and row bytes: Q | K | V, or gate | up) in one launch;
// matrix i writes its rows to columns out_off[i].. of out.
int dc_launch_gemm_tc_multi(dc_ctx* ctx, const dc_weight* const* ws, const int* out_off, int nseg, const uint8_t* act,
                            int n_slots, float* out, int ldo, const int* tile_expert, const int* slot_row, bool accumulate,
                            const int* pair_tile0, const int* pair_nset, int n_pairs) {
    if (nseg < 1 || nseg > 3) return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemm_tc: %d matrices", nseg);
    const dc_weight* w = ws[0];
    GemmTcParams p = {};
    int row_tiles = 0;
    for (int i = 0; i < nseg; ++i) {
        if (!dc_gemm_tc_supports(ws[i])) return dc_fail(ctx, DC_B200_UNSUPPORTED, "gemm_tc: weight type %d or alignment", ws[i]->type);
        if (ws[i]->type != w->type || ws[i]->K != w->K || ws[i]->row_bytes != w->row_bytes || (tile_expert && ws[i]->N != w->N))
            return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemm_tc: matrices of one launch must share type, K and row bytes");
        p.seg[i] = {ws[i]->dev, (int)ws[i]->N, out_off ? out_off[i] : 0};
        row_tiles += ((int)ws[i]->N + TC_ROWS - 1) / TC_ROWS;
    }
    p.nseg = nseg;
    p.row_bytes = (int)w->row_bytes;
    p.K = (int)w->K;
    p.act = act;
    p.n_tt = dc_gemm_tc_tiles(n_slots);
    p.n_slots = n_slots;
    p.out = out;
    p.ldo = ldo;
    p.tile_expert = tile_expert;
    p.slot_row = slot_row;
    p.accumulate = accumulate ? 1 : 0;
    p.estride = (size_t)w->N * w->row_bytes;
    p.one = 1.0f;
    p.err = ctx->d_err;
    if (tile_expert && !pair_tile0) return dc_fail(ctx, DC_B200_INVALID_ARGUMENT, "gemm_tc: grouped matmul without its tile pairs");
    p.pair_tile0 = pair_tile0;
    p.pair_nset = pair_nset;
    p.tiles_x = pair_tile0 ? n_pairs : (p.n_tt + 1) / 2;
    p.tiles_y = row_tiles;
    // one CTA per SM walks its share of the tiles
    const dim3 grid((unsigned)std::min(p.tiles_x * p.tiles_y, ctx->num_sms));
    if (w->type == DC_TYPE_Q4_K) {
        DC_TRY(dc_kernel_setup_unspilled(ctx, (const void*)k_gemm_tc<DC_TYPE_Q4_K>, (int)TC_SMEM, "k_gemm_tc<Q4_K>", TC_LAUNCH_REGS));
        return dc_launch(ctx, "k_gemm_tc", k_gemm_tc<DC_TYPE_Q4_K>, grid, dim3(TC_THREADS), TC_SMEM, p);
    } else {
        DC_TRY(dc_kernel_setup_unspilled(ctx, (const void*)k_gemm_tc<DC_TYPE_Q6_K>, (int)TC_SMEM, "k_gemm_tc<Q6_K>", TC_LAUNCH_REGS));
        return dc_launch(ctx, "k_gemm_tc", k_gemm_tc<DC_TYPE_Q6_K>, grid, dim3(TC_THREADS), TC_SMEM, p);
    }
}

int dc_launch_gemm_tc(dc_ctx* ctx, const dc_weight* w, const uint8_t* act, int n_slots, float* out, int ldo,
                      const int* tile_expert, const int* slot_row, bool accumulate, const int* pair_tile0, const int* pair_nset,
                      int n_pairs) {
    if (pair_tile0)
        return dc_launch_gemm_tc_multi(ctx, &w, nullptr, 1, act, n_slots, out, ldo, tile_expert, slot_row, accumulate, pair_tile0,
                                       pair_nset, n_pairs);
    return dc_launch_gemm_tc_multi(ctx, &w, nullptr, 1, act, n_slots, out, ldo, tile_expert, slot_row, accumulate, nullptr, nullptr, 0);
}
