// Layout of the quantised activations that the tensor-core MUL_MAT reads (gemm_tc.cu), shared with the kernels
// that produce them (prefill.cu).
//
// Per (256-value block, 64-token tile): TC_ACT_TILE bytes = the Q8_K codes as fp16 numbers (exact) in the order of the UMMA's B operand,
// the sums of each token's codes over the block's sixteen 16-value groups as fp16 numbers (exact: at most 16 x 128) as a second B operand, and the
// tile's 64 block scales (f32).
//
// Codes: four quarters of 64 values; a quarter is 64 token rows of 128 bytes, K-major, in 8-row groups of 1024 bytes with the 128-byte swizzle: the
// 16-byte chunk c of row t sits at chunk position c ^ (t % 8) of its row.  Chunk i of a quarter holds values 4 i, 4 i + 2, 4 i + 1, 4 i + 3 of its
// first 32-value sub-block and then the same of its second: the order in which a word of Q4_K nibbles falls apart into fp16 pairs.
// Sums: K-major core matrices of 8 tokens x 16 bytes, the first eight groups of all tokens, then the last eight.
#pragma once
#include <stdint.h>

namespace dc {

constexpr int TC_NTOK = 64;                               // tokens per activation tile
constexpr int TC_QUARTER = TC_NTOK * 128;                 // codes of 64 values of a tile
constexpr int TC_B_Q = 4 * TC_QUARTER;                    // codes of one (block, tile)
constexpr int TC_SUM_HALF = TC_NTOK * 16;                 // sums of eight groups of a tile
constexpr int TC_ACT_SCALES = TC_NTOK * 4;                // the tile's 64 block scales
constexpr int TC_ACT_TILE = TC_B_Q + 2 * TC_SUM_HALF + TC_ACT_SCALES;

// Byte offset, inside a tile's codes, of word w (four codes) of token t's block: 8 bytes.
__host__ __device__ inline uint32_t tc_act_word_offset(int t, int w) {
    const int quarter = w >> 4, chunk = w & 7, second = (w >> 3) & 1;
    return (uint32_t)(quarter * TC_QUARTER + (t >> 3) * 1024 + (t & 7) * 128 + ((chunk ^ (t & 7)) << 4) + 8 * second);
}

#ifdef __CUDACC__
// Four signed bytes as fp16 numbers: bytes 0 and 2, then 1 and 3 (the bits of 1024 + n are 0x6400 + n).
__device__ __forceinline__ uint2 tc_codes_f16(uint32_t w) {
    const uint32_t u = w ^ 0x80808080u;
    const __half2 k = __half2half2(__ushort_as_half(0x6480));      // 1024 + 128
    const uint32_t a = (u & 0x00FF00FFu) | 0x64006400u, b = ((u >> 8) & 0x00FF00FFu) | 0x64006400u;
    const __half2 x = __hsub2(*reinterpret_cast<const __half2*>(&a), k), y = __hsub2(*reinterpret_cast<const __half2*>(&b), k);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
}
// A quantising warp stores token t's block into a tile: lane's 8 codes (w0, w1), the block scale d, and from
// bsum_word (q8k_block_core: the sums of the 16-value group of lanes 2g, 2g+1 and of its neighbour, on every
// lane) the sums.
__device__ __forceinline__ void tc_act_store(uint8_t* tile, int t, int lane, uint32_t w0, uint32_t w1, uint32_t bsum_word,
                                             float d) {
    *reinterpret_cast<uint2*>(tile + tc_act_word_offset(t, 2 * lane)) = tc_codes_f16(w0);
    *reinterpret_cast<uint2*>(tile + tc_act_word_offset(t, 2 * lane + 1)) = tc_codes_f16(w1);
    if ((lane & 3) == 0) {
        const int j = lane >> 2;      // groups 2 j and 2 j + 1
        const __half2 s = __halves2half2(__int2half_rn((int)(int16_t)(bsum_word & 0xFFFFu)), __int2half_rn((int)(int16_t)(bsum_word >> 16)));
        *reinterpret_cast<__half2*>(tile + TC_B_Q + (j >> 2) * TC_SUM_HALF + t * 16 + (j & 3) * 4) = s;
    }
    if (lane == 0) reinterpret_cast<float*>(tile + TC_B_Q + 2 * TC_SUM_HALF)[t] = d;
}
#endif

}  // namespace dc
