// K-quant matrix rows times the Q8_K activations of up to sixteen tokens on the integer tensor instructions
// (mma.sync .s8): the body of k_rows (MUL_MAT) and k_moe_rows (expert rows).
//
// A group of 1, 2, 4 or 8 warps takes a 16-row tile at a time and its super-blocks in turn.  A warp copies the sixteen blocks
// of a unit (tile, super-block) into its own ring in shared memory some units ahead, forms the exact int32 sums of 16 rows x its
// tokens, makes the float terms of the CPU kernels from them and adds these in block order onto sums in registers, so that the
// results are those of the CPU kernels bit for bit.  Where the matrix has too few tiles for one warp each, the warps of a group
// work on neighbouring blocks at the same time, leave their terms in shared memory, and the group's first warp adds them up.
// (Handing the sums on from warp to warp took 240 cycles a block, 2 us of a 16-block row.)
//
// Why integer tensor instructions: one lane decoding a super-block for dp4a (rows_dot) pays the shared-memory reads of the
// activations and a half-rate dp4a per four products for every token and for every row; the fragments of m16n8k32 / m16n8k16 hold
// sixteen rows' codes once for all tokens.  Measured on B200: 8.4 cycles per instruction and scheduler for either shape, against 2
// cycles per dp4a, i.e. 32 to 64 lanes' dp4a in the time of four.
// What bounds it: many rows, issue slots (decoding the codes and the float terms, not the tensor instructions and not the bytes);
// few rows, the latency of a unit's copy and decode, S units of a tile at a time.
// Measured, microseconds at 1 / 4 / 8 / 16 tokens, rows_dot kernels before and these now (bytes alone: 11.5 and 16.8):
//   Q4_K 65536 x 2048   25 / 60 / 158 / 337     22 / 27 / 28 / 40
//   Q6_K 65536 x 2048   53 / 118 / 373 / 743    45 / 59 / 78 / 127
//   Q4_K  6144 x 2048   5.9 for one token       3.7 (rows that it quantises itself)
#pragma once
#include "dc_common.cuh"
#include "dc_internal.h"
#include "dc_stream.cuh"

namespace dc {

#define RW_WARPS 8
#define RW_THREADS (RW_WARPS * 32)
#define RW_STAGES 3           // units in a warp's ring; a fourth would cost an SM its second or third CTA
#define RW_PITCH4 160u        // bytes between a unit's rows, so that 16 lanes' 8-byte loads (4 rows x 32 bytes) fall on distinct banks
#define RW_PITCH6 240u        // the same for 32 lanes' words (8 rows x 16 bytes); 210 bytes at an even offset within the copied 224

// Activation blocks in fragment order (quantize_block_q8f_regs), block-major.
struct RowAct {
    const uint8_t* base;
    int rows;      // capacity
    __device__ __forceinline__ const uint8_t* rec(int b, int row) const { return base + (b * rows + row) * DC_Q8F_BYTES; }
};

struct RowsParams {
    dc_gemv_seg seg[3];
    int n_seg;
    int epi;
    int seg_tiles[3];
    int tiles;                // all segments (expert rows: per expert); Q4_K segments come first
    int tiles4, ctas4;        // tiles of the Q4_K segments, CTAs that work on them
    int S;                    // warps of a group
    uint32_t stage_bytes;
    uint32_t off_zero, off_link, off_ring;
    const uint8_t* act_q8;
    const float* act_f32;     // given: the rows still to be quantised, which every CTA does for its own
    const float* norm_w;      // given: and to be normed before that
    float norm_eps;
    int T, K, nb;
    int act_rows;             // rows of activations a CTA holds
    unsigned long long* argmax;
    BlockSumDump dump;
    // expert rows
    const uint8_t *w0, *w1;
    int type, row_bytes, N, top_k, e_base;
    const int *n_active;
    const int32_t *uexp, *uoff, *uassign;
    float* out;
};

__device__ __forceinline__ void mma_k32_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_k32_u8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_k16_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ uint32_t ld_w(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ float ld_f(const uint8_t* p) { return *reinterpret_cast<const float*>(p); }
__device__ __forceinline__ uint4 ld_v4(const uint8_t* p) { return *reinterpret_cast<const uint4*>(p); }
// byte k of a word, unsigned / signed
template <int K>
__device__ __forceinline__ int byte_u(uint32_t w) { return (int)__byte_perm(w, 0, 0x4440 + K); }
template <int K>
__device__ __forceinline__ int byte_s(uint32_t w) {
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "n"(0x8880 + 0x1111 * K));
    return (int)r;
}
// 32 bits from a 2-byte aligned address, given as the aligned one and 0 or 16
__device__ __forceinline__ uint32_t ld_w2(const uint8_t* p4, uint32_t shift) { return __funnelshift_r(ld_w(p4), ld_w(p4 + 4), shift); }

// One Q4_K super-block of 16 rows (this lane: rows g and g + 8 at rg, rg8) against block b of tokens row0 .. row0 + nt - 1; the two
// terms of sum i (four per eight tokens) go to sink(i, I term, M term).  Sub-block s times its tokens' codes is one m16n8k32; its sums enter I times the sub-block's scale.
// High nibbles stay in place (bytes 16 q, unsigned), so that their sums are 16 times the wanted ones, exactly.  The minimum term is
// two more products over the eight 32-value sums, whose low and high bytes are separate operands.
// ONE: a single token, column 0 alone.
template <int NG, bool ONE, bool DUMP, class Sink>
__device__ __forceinline__ void rows_unit_q4k(const uint8_t* rg, const uint8_t* rg8, const RowAct& act, int b, int row0, int nt, int lane,
                                              const RowsParams& p, int row, bool live, bool live8, const Sink& sink) {
    const int g = lane >> 2, t = lane & 3;
    const uint4 h = ld_v4(rg), h8 = ld_v4(rg8);
    uint32_t w[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int o = 16 + 32 * c + 8 * t;
        const uint2 x = *reinterpret_cast<const uint2*>(rg + o), y = *reinterpret_cast<const uint2*>(rg8 + o);
        w[c][0] = x.x;
        w[c][1] = y.x;
        w[c][2] = x.y;
        w[c][3] = y.y;
    }
    const uint32_t sc[2] = {h.y & 0x3f3f3f3fu, (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u)};
    const uint32_t sc8[2] = {h8.y & 0x3f3f3f3fu, (h8.w & 0x0f0f0f0fu) | ((h8.y >> 2) & 0x30303030u)};
    // threads 0 and 1 of a group: the minima of sub-blocks 0..3, 4..7; the others' operands are zero
    const uint32_t keep = t < 2 ? 0x3f3f3f3fu : 0u;
    const uint32_t m = (t ? ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u) : h.z) & keep;
    const uint32_t m8 = (t ? ((h8.w >> 4) & 0x0f0f0f0fu) | ((h8.z >> 2) & 0x30303030u) : h8.z) & keep;
    const float d0 = fp16_bits_to_float((uint16_t)(h.x & 0xFFFF)), dm0 = fp16_bits_to_float((uint16_t)(h.x >> 16));
    const float d8 = fp16_bits_to_float((uint16_t)(h8.x & 0xFFFF)), dm8 = fp16_bits_to_float((uint16_t)(h8.x >> 16));
#pragma unroll
    for (int tg = 0; tg < NG; ++tg) {
        if (tg && 8 * tg >= nt) break;
        const uint8_t* rec = act.rec(b, row0 + min(8 * tg + g, nt - 1));
        int lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0}, ml[4], mh[4];
        mma_k16_s8(ml, m, m8, ld_w(rec + 64 + 4 * (t & 1)));
        mma_k16_s8(mh, m, m8, ld_w(rec + 72 + 4 * (t & 1)));
        rec += 160 * (t & 1) + 16 * (t >> 1);      // words 2 t and 2 t + 1 of every sub-block: two runs, one of their groups
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint4 q0 = ld_v4(rec + 32 * j), q1 = ld_v4(rec + 32 * j + 80);   // quadrants of the half: the first word, the second
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t* x = w[2 * j + k];
                int d[4];
                mma_k32_s8(d, x[0] & 0x0F0F0F0Fu, x[1] & 0x0F0F0F0Fu, x[2] & 0x0F0F0F0Fu, x[3] & 0x0F0F0F0Fu, k ? q0.z : q0.x, k ? q1.z : q1.x);
                int a = k ? byte_u<2>(sc[j]) : byte_u<0>(sc[j]), a8 = k ? byte_u<2>(sc8[j]) : byte_u<0>(sc8[j]);
                lo[0] += a * d[0];
                lo[2] += a8 * d[2];
                if (!ONE) {
                    lo[1] += a * d[1];
                    lo[3] += a8 * d[3];
                }
                mma_k32_u8(d, x[0] & 0xF0F0F0F0u, x[1] & 0xF0F0F0F0u, x[2] & 0xF0F0F0F0u, x[3] & 0xF0F0F0F0u, k ? q0.w : q0.y, k ? q1.w : q1.y);
                a = k ? byte_u<3>(sc[j]) : byte_u<1>(sc[j]), a8 = k ? byte_u<3>(sc8[j]) : byte_u<1>(sc8[j]);
                hi[0] += a * d[0];
                hi[2] += a8 * d[2];
                if (!ONE) {
                    hi[1] += a * d[1];
                    hi[3] += a8 * d[3];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < (ONE ? 1 : 2); ++k) {
            const float yd = ld_f(act.rec(b, row0 + min(8 * tg + 2 * t + k, nt - 1)) + 144);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int i = 2 * r + k, I = lo[i] + (hi[i] >> 4), M = ml[i] + 256 * mh[i];
                sink(4 * tg + i, __fmul_rn(__fmul_rn(r ? d8 : d0, yd), (float)I), __fmul_rn(__fmul_rn(r ? dm8 : dm0, yd), (float)M));
                if (DUMP && 8 * tg + 2 * t + k < nt && (r ? live8 : live)) {
                    const size_t at = ((size_t)(8 * tg + 2 * t + k) * p.dump.N + row + 8 * r) * p.nb + b;
                    p.dump.I[at] = I;
                    if (p.dump.M) p.dump.M[at] = M;
                }
            }
        }
    }
}

// Four codes 4 (q - 32) as signed bytes, from words whose bytes hold the low four bits of q at bits 2..5 and the upper two at bits
// 6..7: 4 q with the top bit flipped.  (q - 32 itself takes two instructions more; the sums are shifted down, exactly.)
__device__ __forceinline__ uint32_t rows_q6x4(uint32_t lo, uint32_t hi) { return (lo & 0x3C3C3C3Cu) | ((hi & 0xC0C0C0C0u) ^ 0x80808080u); }

// One Q6_K super-block of 16 rows (2-byte aligned) against block b of up to 2 NP tokens; partial i (eight per two
// tokens) and its factor go to sink(i, P, f).  The CPU kernel
// keeps eight int32 partials per block: partial L collects bytes 4 (L % 4) .. + 3 of the 16-value groups L / 4, L / 4 + 2, ... times the
// groups' scales.  So the four words of a group must not be added up: an m16n8k16 takes one group of 16 rows, and its eight columns are
// the four words of two tokens, the others' codes being zero in each column (a lane whose column is not its word reads zeros).
template <int NP, bool DUMP, class Sink>
__device__ __forceinline__ void rows_unit_q6k(const uint8_t* smem, uint32_t og, uint32_t og8, const RowAct& act, int b, int row0, int nt, int lane,
                                              const RowsParams& p, int row, bool live, bool live8, const Sink& sink) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t sh = (og & 2u) * 8u, sh8 = (og8 & 2u) * 8u;
    const uint8_t *a = smem + (og & ~3u), *a8 = smem + (og8 & ~3u);
    // the block scale lies at the block's byte 208, in the word at 208 or across that word's upper half
    const float d0 = fp16_bits_to_float((uint16_t)(ld_w(a + 208) >> sh)), d8 = fp16_bits_to_float((uint16_t)(ld_w(a8 + 208) >> sh8));
    uint32_t sc[4], sc8[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sc[i] = ld_w2(a + 192 + 4 * i, sh);
        sc8[i] = ld_w2(a8 + 192 + 4 * i, sh8);
    }
    int total[NP][2];
#pragma unroll
    for (int wq = 0; wq < 2; ++wq) {      // partials 0..3, then 4..7: half of the decoded codes live at a time
        uint32_t q[2][4][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint8_t* base = (r ? a8 : a) + 16 * wq + 4 * t;
                const uint32_t s = r ? sh8 : sh;
                const uint32_t la = ld_w2(base + 64 * j, s), lc = ld_w2(base + 64 * j + 32, s), lh = ld_w2(base + 128 + 32 * j, s);
                q[j][0][r] = rows_q6x4(la << 2, lh << 6);
                q[j][1][r] = rows_q6x4(lc << 2, lh << 4);
                q[j][2][r] = rows_q6x4(la >> 2, lh << 2);
                q[j][3][r] = rows_q6x4(lc >> 2, lh);
            }
#pragma unroll
        for (int pr = 0; pr < NP; ++pr) {
            if (pr && 2 * pr >= nt) break;
            const int mine = 2 * pr + (g >> 2);
            const uint8_t* src = smem + ((g & 3) == t && mine < nt ? (uint32_t)((b * act.rows + row0 + mine) * DC_Q8F_BYTES + 80 * t) : p.off_zero);
            int P[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint4 y = ld_v4(src + 32 * j + 16 * wq);
#pragma unroll
                for (int qd = 0; qd < 4; ++qd) {
                    int d[4];
                    mma_k16_s8(d, q[j][qd][0], q[j][qd][1], qd == 0 ? y.x : qd == 1 ? y.y : qd == 2 ? y.z : y.w);
                    const uint32_t w0 = sc[2 * j + (qd >> 1)], w8 = sc8[2 * j + (qd >> 1)];
                    const int at = 2 * (qd & 1) + wq;
                    const int s0 = at == 0 ? byte_s<0>(w0) : at == 1 ? byte_s<1>(w0) : at == 2 ? byte_s<2>(w0) : byte_s<3>(w0);
                    const int s8 = at == 0 ? byte_s<0>(w8) : at == 1 ? byte_s<1>(w8) : at == 2 ? byte_s<2>(w8) : byte_s<3>(w8);
                    P[0] += s0 * d[0];
                    P[1] += s0 * d[1];
                    P[2] += s8 * d[2];
                    P[3] += s8 * d[3];
                }
            }
            const int tok = min(2 * pr + (t >> 1), nt - 1);
            const float yd = ld_f(act.rec(b, row0 + tok) + 144), f0 = __fmul_rn(yd, d0), f8 = __fmul_rn(yd, d8);
            if (DUMP) {
                total[pr][0] = (wq ? total[pr][0] : 0) + (P[0] >> 2) + (P[1] >> 2);
                total[pr][1] = (wq ? total[pr][1] : 0) + (P[2] >> 2) + (P[3] >> 2);
                const int s0 = total[pr][0] + __shfl_xor_sync(0xffffffffu, total[pr][0], 1), s8 = total[pr][1] + __shfl_xor_sync(0xffffffffu, total[pr][1], 1);
                if (wq && (t & 1) == 0 && 2 * pr + (t >> 1) < nt) {
                    const size_t at = ((size_t)tok * p.dump.N + row) * p.nb + b;
                    if (live) p.dump.I[at] = s0;
                    if (live8) p.dump.I[at + 8 * (size_t)p.nb] = s8;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) sink(8 * pr + 4 * wq + i, (float)(P[i] >> 2), i < 2 ? f0 : f8);
        }
    }
}

// The same for a single token on m16n8k32: a 32-value quadrant of 16 rows at a time, whose eight words are the eight columns and
// partials, so that a lane's two columns have one scale.
template <bool DUMP, class Sink>
__device__ __forceinline__ void rows_unit_q6k_one(const uint8_t* smem, uint32_t og, uint32_t og8, const RowAct& act, int b, int row0, int lane,
                                                  const RowsParams& p, int row, bool live, bool live8, const Sink& sink) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t sh = (og & 2u) * 8u, sh8 = (og8 & 2u) * 8u;
    const uint8_t *a = smem + (og & ~3u), *a8 = smem + (og8 & ~3u);
    const float d0 = fp16_bits_to_float((uint16_t)(ld_w(a + 208) >> sh)), d8 = fp16_bits_to_float((uint16_t)(ld_w(a8 + 208) >> sh8));
    const uint32_t rec = (uint32_t)((b * act.rows + row0) * DC_Q8F_BYTES);
    const uint8_t* y0 = smem + (g == t ? rec + 80 * t : p.off_zero);
    const uint8_t* y1 = smem + (g == t + 4 ? rec + 80 * t : p.off_zero);
    const uint32_t which = 8u * (t >> 1);       // columns 2 t and 2 t + 1 lie in group t / 2 of the quadrant
    int P[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        uint32_t q[2][4][2];
#pragma unroll
        for (int wq = 0; wq < 2; ++wq)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint8_t* base = (r ? a8 : a) + 16 * wq + 4 * t;
                const uint32_t s = r ? sh8 : sh;
                const uint32_t la = ld_w2(base + 64 * j, s), lc = ld_w2(base + 64 * j + 32, s), lh = ld_w2(base + 128 + 32 * j, s);
                q[wq][0][r] = rows_q6x4(la << 2, lh << 6);
                q[wq][1][r] = rows_q6x4(lc << 2, lh << 4);
                q[wq][2][r] = rows_q6x4(la >> 2, lh << 2);
                q[wq][3][r] = rows_q6x4(lc >> 2, lh);
            }
        const uint4 b0 = ld_v4(y0 + 32 * j), b1 = ld_v4(y1 + 32 * j + 16);
        uint32_t sc[2], sc8[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            sc[i] = ld_w2(a + 192 + 8 * j + 4 * i, sh) >> which;
            sc8[i] = ld_w2(a8 + 192 + 8 * j + 4 * i, sh8) >> which;
        }
#pragma unroll
        for (int qd = 0; qd < 4; ++qd) {
            int d[4];
            mma_k32_s8(d, q[0][qd][0], q[0][qd][1], q[1][qd][0], q[1][qd][1], qd == 0 ? b0.x : qd == 1 ? b0.y : qd == 2 ? b0.z : b0.w,
                       qd == 0 ? b1.x : qd == 1 ? b1.y : qd == 2 ? b1.z : b1.w);
            const int s0 = qd & 1 ? byte_s<2>(sc[qd >> 1]) : byte_s<0>(sc[qd >> 1]), s8 = qd & 1 ? byte_s<2>(sc8[qd >> 1]) : byte_s<0>(sc8[qd >> 1]);
            P[0] += s0 * d[0];
            P[1] += s0 * d[1];
            P[2] += s8 * d[2];
            P[3] += s8 * d[3];
        }
    }
    if (DUMP) {
        int s0 = (P[0] >> 2) + (P[1] >> 2), s8 = (P[2] >> 2) + (P[3] >> 2);
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            s8 += __shfl_xor_sync(0xffffffffu, s8, o);
        }
        if (t == 0 && live) p.dump.I[(size_t)row * p.nb + b] = s0;
        if (t == 0 && live8) p.dump.I[(size_t)(row + 8) * p.nb + b] = s8;
    }
    const float yd = ld_f(smem + rec + 144), f0 = __fmul_rn(yd, d0), f8 = __fmul_rn(yd, d8);
#pragma unroll
    for (int i = 0; i < 4; ++i) sink(i, (float)(P[i] >> 2), i < 2 ? f0 : f8);
}

struct RowsTile {
    const uint8_t *w, *w_up;   // first row; w_up: the up rows of a gate/up pair
    int row_bytes;
    int row0, rows;
    float* out;
    int ldo;
    int a0, nt;                // expert rows: first assignment, tokens of the expert
};

template <bool MOE>
__device__ __forceinline__ RowsTile rows_tile(const RowsParams& p, int i) {
    RowsTile r;
    if (MOE) {
        const int u = i / p.tiles, k = i - u * p.tiles;
        r.row_bytes = p.row_bytes;
        r.row0 = 16 * k;
        r.rows = min(16, p.N - r.row0);
        const size_t off = ((size_t)(p.uexp[u] - p.e_base) * p.N + r.row0) * p.row_bytes;
        r.w = p.w0 + off;
        r.w_up = p.w1 ? p.w1 + off : nullptr;
        r.a0 = p.uoff[u];
        r.nt = p.uoff[u + 1] - r.a0;
        r.out = p.out;
        r.ldo = p.N;
    } else {
        int s = 0;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (s == k && k + 1 < p.n_seg && i >= p.seg_tiles[k]) {
                i -= p.seg_tiles[k];
                s = k + 1;
            }
        const dc_gemv_seg g = s == 0 ? p.seg[0] : s == 1 ? p.seg[1] : p.seg[2];
        r.row_bytes = g.row_bytes;
        r.row0 = 16 * i;
        r.rows = min(16, g.n_rows - r.row0);
        r.w = g.w + (size_t)r.row0 * g.row_bytes;
        r.w_up = p.epi == DC_EPI_SWIGLU ? p.seg[1].w + (size_t)r.row0 * g.row_bytes : nullptr;
        r.a0 = 0;
        r.nt = p.T;
        r.out = g.out;
        r.ldo = g.ldo;
    }
    return r;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The norm weights of a warp's first block, fetched while the kernel still waits for its predecessor: they are older than this step and
// as a rule no longer in L2.  With the rows' values kept in registers between the sum of squares and the quantiser: a dense decode step of
// 28 layers 1.6 % shorter.
struct RowsNormW {
    float4 a, b;
    __device__ __forceinline__ void fetch(const RowsParams& p) {
        a = b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!p.norm_w) return;
        const float4* w = reinterpret_cast<const float4*>(p.norm_w + (threadIdx.x >> 5) % p.nb * DC_QK_K) + 2 * (threadIdx.x & 31);
        a = w[0];
        b = w[1];
    }
};

// Blocks [0, nb) of `n` activation rows into shared memory; row i of the CTA's list is row src(i) of the quantised rows.
// NORM: p.norm_w may be given.
template <bool NORM, class Src>
__device__ __forceinline__ void rows_fill_act(const RowsParams& p, uint8_t* smem, int n, const RowsNormW& nw, const Src& src) {
    constexpr int PIECES = DC_Q8F_BYTES / 16;
    const int nb = p.nb, rows = p.act_rows;
    if (NORM && p.norm_w) {      // few rows (dc_rows_quantise), a block of 256 values to a warp: k_rmsnorm_q8k's arithmetic
        __shared__ double s_ss[24];      // the blocks' sums of squares
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const float4* x = reinterpret_cast<const float4*>(p.act_f32) + 2 * lane;
        float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
        // the first block last: it stays in registers
        for (int i = (n * nb - 1 - warp) / RW_WARPS * RW_WARPS + warp; i >= 0 && i < n * nb; i -= RW_WARPS) {
            x0 = __ldcg(x + i * (DC_QK_K / 4));
            x1 = __ldcg(x + i * (DC_QK_K / 4) + 1);
            double ss = (((double)x0.x * x0.x + (double)x0.y * x0.y) + ((double)x0.z * x0.z + (double)x0.w * x0.w)) +
                        (((double)x1.x * x1.x + (double)x1.y * x1.y) + ((double)x1.z * x1.z + (double)x1.w * x1.w));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) s_ss[i] = ss;
        }
        __syncthreads();
        float4 w0 = nw.a, w1 = nw.b;
        for (int i = warp; i < n * nb; i += RW_WARPS) {
            const int row = i / nb, b = i - row * nb;
            if (i != warp) {
                x0 = __ldcg(x + i * (DC_QK_K / 4));
                x1 = __ldcg(x + i * (DC_QK_K / 4) + 1);
                const float4* w = reinterpret_cast<const float4*>(p.norm_w + b * DC_QK_K) + 2 * lane;
                w0 = w[0];
                w1 = w[1];
            }
            double tot = 0.0;
            for (int k = 0; k < nb; ++k) tot += s_ss[row * nb + k];
            const float mean = (float)(tot / (double)p.K);
            const float f = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, p.norm_eps)));
            const float v[8] = {__fmul_rn(__fmul_rn(x0.x, f), w0.x), __fmul_rn(__fmul_rn(x0.y, f), w0.y), __fmul_rn(__fmul_rn(x0.z, f), w0.z), __fmul_rn(__fmul_rn(x0.w, f), w0.w),
                                __fmul_rn(__fmul_rn(x1.x, f), w1.x), __fmul_rn(__fmul_rn(x1.y, f), w1.y), __fmul_rn(__fmul_rn(x1.z, f), w1.z), __fmul_rn(__fmul_rn(x1.w, f), w1.w)};
            quantize_block_q8f_regs(v, smem + (b * rows + row) * DC_Q8F_BYTES, lane);
        }
        return;
    }
    if (p.act_f32) {
        for (int i = threadIdx.x >> 5; i < n * nb; i += RW_WARPS) {
            const int row = i / nb, b = i - row * nb;
            quantize_block_q8k_warp<true>(p.act_f32 + ((size_t)src(row) * nb + b) * DC_QK_K, smem + (b * rows + row) * DC_Q8F_BYTES, threadIdx.x & 31);
        }
        return;
    }
    const uint32_t base = smem_u32(smem);
    for (int i = threadIdx.x; i < n * nb * PIECES; i += RW_THREADS) {
        const int blk = i / PIECES, o = 16 * (i - blk * PIECES), row = blk / nb, b = blk - row * nb;
        cp_async16(base + (uint32_t)(b * rows + row) * DC_Q8F_BYTES + o, p.act_q8 + ((size_t)src(row) * nb + b) * DC_Q8F_BYTES + o);
    }
}

// The units that a warp copies: for every tile of its group, for the gate and then the up rows of a pair, blocks w, w + S, ...  s0, s1: this lane's rows g and g + 8 of the unit in global memory (rows past the matrix's
// end are read as its last row, their sums are not stored).
template <int TYPE, bool MOE, bool PAIR>
struct RowsWalk {
    static constexpr int BB = TYPE == DC_TYPE_Q4_K ? DC_Q4K_BYTES : DC_Q6K_BYTES;
    int i, end, step;      // tile of the list
    int b, up;
    const uint8_t *s0, *s1;
    RowsTile t;
    bool valid;
    __device__ __forceinline__ void rows(int g) {
        const uint8_t* w = (PAIR && up ? t.w_up : t.w) + b * BB;
        s0 = w + (size_t)min(g, t.rows - 1) * t.row_bytes;
        s1 = w + (size_t)min(g + 8, t.rows - 1) * t.row_bytes;
    }
    __device__ __forceinline__ void start(const RowsParams& p, int first, int end_, int step_, int w, int g) {
        i = first;
        end = end_;
        step = step_;
        b = w;
        up = 0;
        valid = i < end;
        if (valid) {
            t = rows_tile<MOE>(p, i);
            rows(g);
        }
    }
    __device__ __forceinline__ void next(const RowsParams& p, int S, int w, int g) {
        b += S;
        if (b < p.nb) {
            s0 += S * BB;
            s1 += S * BB;
            return;
        }
        b = w;
        if (PAIR && !up) {
            up = 1;
        } else {
            up = 0;
            i += step;
            valid = i < end;
            if (!valid) return;
            t = rows_tile<MOE>(p, i);
        }
        rows(g);
    }
};

// Four lanes copy a row: 9 or 14 pieces of 16 bytes.
template <int TYPE>
__device__ __forceinline__ void rows_copy(const uint8_t* s, uint32_t d, int t) {
    d += 16 * t;
    if (TYPE == DC_TYPE_Q4_K) {
        s += 16 * t;
        cp_async16(d, s);
        cp_async16(d + 64, s + 64);
        if (t == 0) cp_async16(d + 128, s + 128);
    } else {
        const int skew = (int)((uintptr_t)s & 15), n = (skew + DC_Q6K_BYTES + 15) & ~15;
        s = s - skew + 16 * t;
        cp_async16(d, s);
        cp_async16(d + 64, s + 64);
        cp_async16(d + 128, s + 128);
        if (192 + 16 * t < n) cp_async16(d + 192, s + 192);
    }
}

// The whole CTA on tiles [lo, hi) of a list, of which this is CTA `cta` of `ctas`; NP: pairs of tokens.  PREFETCH: the rows to read are
// known before the predecessor's results are (a product's always are, an expert's where the routing is older than the predecessor).
template <int TYPE, int NP, bool ONE, bool ALONE, bool MOE, bool PAIR, bool DUMP, bool PREFETCH>
__device__ __forceinline__ void rows_cta(const RowsParams& p, uint8_t* smem, int cta, int ctas, int lo, int hi) {
    constexpr bool Q4 = TYPE == DC_TYPE_Q4_K;
    constexpr int NS = RW_STAGES, NG = (NP + 3) / 4, NA = Q4 || ONE ? 4 * NG : 8 * NP, NR = Q4 ? 4 * NG : 2 * NP;   // sums, results of a lane
    constexpr uint32_t PITCH = Q4 ? RW_PITCH4 : RW_PITCH6, STAGE = 16 * PITCH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const uint32_t sm = smem_u32(smem);
    if (threadIdx.x < 16) reinterpret_cast<uint32_t*>(smem + p.off_zero)[threadIdx.x] = 0u;
    // a gate/up kernel of experts lets its successor start only when the routing is final: that one reads it before its own wait
    if (PREFETCH) pdl_launch_dependents();
    if (!PREFETCH) {
        pdl_wait();
        pdl_launch_dependents();
    }
    // expert rows: neighbouring tiles, so that a CTA meets few experts' tokens; matrices: tiles in turn
    const int S = ALONE ? 1 : p.S, groups = RW_WARPS / S, w = warp & (S - 1), grp = warp / S;      // ALONE: groups of one warp
    int first, end, step;
    if (MOE) {
        const unsigned total = (unsigned)(*p.n_active) * (unsigned)p.tiles;
        first = (int)((unsigned long long)total * cta / ctas);
        end = (int)((unsigned long long)total * (cta + 1) / ctas);
        step = groups;
    } else {
        first = lo + cta * groups;
        end = hi;
        step = ctas * groups;
    }
    const bool works = w < p.nb;     // a group may have more warps than the row has blocks
    const uint32_t ring = p.off_ring + (uint32_t)warp * NS * STAGE;
    RowsWalk<TYPE, MOE, PAIR> prod;
    prod.start(p, first + grp, works ? end : 0, step, w, g);
    auto copy = [&](uint32_t slot) {
        const uint32_t d = sm + ring + slot * STAGE + g * PITCH;
        rows_copy<TYPE>(prod.s0, d, tq);
        rows_copy<TYPE>(prod.s1, d + 8 * PITCH, tq);
    };
    uint32_t head = 0;
#pragma unroll 1
    for (int s = 0; s < NS - 1; ++s) {
        if (prod.valid) {
            copy(head);
            prod.next(p, S, w, g);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        ++head;
    }
    RowsNormW nw = {};
    if (!MOE) nw.fetch(p);      // (expert rows come normed)
    if (PREFETCH) pdl_wait();
    const RowAct act = {smem, p.act_rows};
    int a_lo = 0;
    if (MOE) {
        if (first < end) {
            const int u0 = first / p.tiles, u1 = (end - 1) / p.tiles;
            a_lo = p.uoff[u0];
            const int32_t* list = p.uassign + a_lo;
            const int per = PAIR ? p.top_k : 1;
            rows_fill_act<false>(p, smem, min(p.uoff[u1 + 1] - a_lo, p.act_rows), nw, [=](int i) { return list[i] / per; });
        }
    } else {
        rows_fill_act<true>(p, smem, p.T, nw, [](int i) { return i; });
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    cp_async_wait<0>();
    __syncthreads();
    // terms of a group's warps, two floats a sum (Q4_K: I and M term; Q6_K: partial, and one factor per four of them)
    constexpr int NT = Q4 ? 2 * NA : NA + NA / 2;
    float* own = reinterpret_cast<float*>(smem + p.off_link) + warp * NT * 32 + lane;
    const float* all = reinterpret_cast<const float*>(smem + p.off_link) + grp * S * NT * 32 + lane;
    uint32_t tail = 0;
    unsigned long long best[NR];      // largest result so far of every token that the lane holds (rows g and g + 8 share one)
#pragma unroll
    for (int i = 0; i < NR; ++i) best[i] = 0ull;
    float acc[NA], gate[PAIR ? NR : 1] = {};
    auto add = [&](int i, float x, float y) {
        if (Q4) acc[i] = __fsub_rn(__fadd_rn(acc[i], x), y);
        else acc[i] = __fmaf_rn(y, x, acc[i]);
    };
    auto sink = [&](int i, float x, float y) {
        if (ALONE) {
            add(i, x, y);
        } else if (Q4) {
            own[(2 * i) * 32] = x;
            own[(2 * i + 1) * 32] = y;
        } else {
            own[i * 32] = x;
            if ((i & 1) == 0 && (ONE || (i & 4) == 0)) own[(NA + (ONE ? i >> 1 : (i >> 3) * 2 + (i >> 1 & 1))) * 32] = y;
        }
    };
    auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * S) : "memory"); };
    for (int tile = first + grp; tile < end; tile += step) {
        const RowsTile t = rows_tile<MOE>(p, tile);
        const int nt = ONE ? 1 : t.nt, row0 = t.a0 - a_lo;
        for (int up = 0; up < (PAIR ? 2 : 1); ++up) {
#pragma unroll
            for (int i = 0; i < NA; ++i) acc[i] = 0.0f;
            // where in its first 16-byte piece a row's block 0 starts (Q6_K)
            const uint32_t sk0 = (uint32_t)(uintptr_t)((PAIR && up ? t.w_up : t.w) + (size_t)min(g, t.rows - 1) * t.row_bytes);
            const uint32_t sk8 = (uint32_t)(uintptr_t)((PAIR && up ? t.w_up : t.w) + (size_t)min(g + 8, t.rows - 1) * t.row_bytes);
            for (int b0 = 0; b0 < p.nb; b0 += S) {
                const int b = b0 + w;
                if (b < p.nb) {
                    if (prod.valid) {
                        copy(head);
                        prod.next(p, S, w, g);
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    head = head + 1 == NS ? 0 : head + 1;
                    cp_async_wait<NS - 1>();
                    __syncwarp();
                    const uint32_t stage = ring + tail * STAGE + g * PITCH;
                    if constexpr (Q4)
                        rows_unit_q4k<NG, ONE, DUMP>(smem + stage, smem + stage + 8 * PITCH, act, b, row0, nt, lane, p, t.row0 + g, g < t.rows, g + 8 < t.rows, sink);
                    else if constexpr (ONE)
                        rows_unit_q6k_one<DUMP>(smem, stage + (sk0 + b * DC_Q6K_BYTES & 15u), stage + 8 * PITCH + (sk8 + b * DC_Q6K_BYTES & 15u), act, b, row0, lane, p,
                                                t.row0 + g, g < t.rows, g + 8 < t.rows, sink);
                    else
                        rows_unit_q6k<NP, DUMP>(smem, stage + (sk0 + b * DC_Q6K_BYTES & 15u), stage + 8 * PITCH + (sk8 + b * DC_Q6K_BYTES & 15u), act, b, row0, nt, lane, p,
                                                t.row0 + g, g < t.rows, g + 8 < t.rows, sink);
                    __syncwarp();
                    tail = tail + 1 == NS ? 0 : tail + 1;
                }
                if (ALONE) continue;
                meet();
                if (w == 0) {
                    const int n = min(S, p.nb - b0);
#pragma unroll 2
                    for (int k = 0; k < n; ++k) {
                        const float* x = all + k * NT * 32;
#pragma unroll
                        for (int i = 0; i < NA; ++i) {
                            if (Q4 ? (ONE && (i & 1)) || (i >= 4 && 8 * (i >> 2) >= nt) : !ONE && 2 * (i >> 3) >= nt) continue;
                            if (Q4) add(i, x[(2 * i) * 32], x[(2 * i + 1) * 32]);
                            else add(i, x[i * 32], x[(NA + (ONE ? i >> 1 : (i >> 3) * 2 + (i >> 1 & 1))) * 32]);
                        }
                    }
                }
                meet();      // the terms have been read
            }
            if (w != 0) continue;
            // result i: Q4_K: token 8 (i / 4) + 2 tq + i % 2, row g + 8 (i / 2 % 2); Q6_K: token 2 (i / 2) + tq / 2, row g + 8 (i % 2)
            float v[NR];
            if constexpr (Q4) {
#pragma unroll
                for (int i = 0; i < NR; ++i) v[i] = acc[i];
            } else {
                // a single token: lane t of four holds partials 2 t and 2 t + 1; else lane pairs hold 0, 1, 4, 5 and 2, 3, 6, 7 of a token
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    if (ONE) {
                        const float x0 = __fadd_rn(acc[2 * i], __shfl_xor_sync(0xffffffffu, acc[2 * i], 2)), x1 = __fadd_rn(acc[2 * i + 1], __shfl_xor_sync(0xffffffffu, acc[2 * i + 1], 2));
                        v[i] = __fadd_rn(__fadd_rn(x0, __shfl_xor_sync(0xffffffffu, x0, 1)), __fadd_rn(x1, __shfl_xor_sync(0xffffffffu, x1, 1)));
                        continue;
                    }
                    const float* c = acc + 8 * (i >> 1) + 2 * (i & 1);
                    const float x0 = __fadd_rn(c[0], c[4]), x1 = __fadd_rn(c[1], c[5]);
                    v[i] = __fadd_rn(__fadd_rn(x0, __shfl_xor_sync(0xffffffffu, x0, 1)), __fadd_rn(x1, __shfl_xor_sync(0xffffffffu, x1, 1)));
                }
            }
            if (PAIR && !up) {
#pragma unroll
                for (int i = 0; i < NR; ++i) gate[i] = v[i];
                continue;
            }
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int tok = Q4 ? 8 * (i >> 2) + 2 * tq + (i & 1) : 2 * (i >> 1) + (tq >> 1), r = Q4 ? i >> 1 & 1 : i & 1;
                if (tok >= nt || g + 8 * r >= t.rows || (!Q4 && (tq & 1) != r) || (Q4 && ONE && (i & 1))) continue;     // one lane of a Q6_K pair stores each row
                const int row = t.row0 + g + 8 * r;
                const float x = PAIR ? __fmul_rn(silu_fast(gate[i]), v[i]) : v[i];
                if (MOE) {
                    t.out[(size_t)p.uassign[t.a0 + tok] * t.ldo + row] = x;
                } else {
                    float* o = t.out + (size_t)tok * t.ldo + row;
                    *o = p.epi == DC_EPI_ACC ? __ldcg(o) + x : x;   // L2 read: another SM may have written it
                    if (p.argmax) {
                        const unsigned long long key = argmax_key(x, row);
                        unsigned long long& top = best[Q4 ? i & ~2 : i & ~1];
                        top = key > top ? key : top;
                    }
                }
            }
        }
    }
    cp_async_wait<0>();
    if (!MOE && p.argmax) {
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            if (Q4 ? i & 2 : i & 1) continue;
            unsigned long long k = best[i];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                if (o == 2 || (Q4 && o == 1)) continue;      // another token's lane
                const unsigned long long ok = __shfl_xor_sync(0xffffffffu, k, o);
                k = ok > k ? ok : k;
            }
            const int tok = Q4 ? 8 * (i >> 2) + 2 * tq + (i & 1) : 2 * (i >> 1) + (tq >> 1);
            if (g == 0 && (Q4 || !(tq & 1)) && k && tok < p.T) atomicMax(p.argmax + tok, k);
        }
    }
}

// Sizes of a launch; returns the dynamic shared memory, or 0 if the activations leave no room.  S: as many warps a tile as keep the SMs'
// warps (two or three CTAs of eight) busy, for the tiles then run at the same time and a tile's latency is a few blocks' instead of all of them.
// Above that line every warp has a tile of its own and the terms stay in registers: 65536 x 2048, 16 tokens, Q4_K 40 us against 46, and
// Q6_K 127 against 143, for a kernel that also carries the code of the shared terms.
static inline size_t rows_plan(RowsParams& p, int np, bool has_q6, long long tiles, int num_sms) {
    const long long warps = (has_q6 ? 16ll : 24ll) * num_sms;
    p.S = 1;
    while (p.S < RW_WARPS && p.S < p.nb && tiles * p.S * 2 <= warps) p.S *= 2;
    p.stage_bytes = 16 * (has_q6 ? RW_PITCH6 : RW_PITCH4);
    auto size = [&]() {
        p.off_zero = (uint32_t)((size_t)p.act_rows * p.nb * DC_Q8F_BYTES);
        p.off_link = p.off_zero + 128;
        p.off_ring = p.off_link + (p.S > 1 ? (uint32_t)(RW_WARPS * 12 * np * 32 * 4) : 0u);
        return (size_t)p.off_ring + (size_t)RW_WARPS * RW_STAGES * p.stage_bytes;
    };
    if (size() > 220 * 1024) p.S = 1;
    const size_t total = size();
    return total <= 220 * 1024 ? total : 0;
}

}  // namespace dc
