// hx_digits.cuh -- f32 values as base-13 digit columns for the FP4 tensor cores: the table and the conversion that k_pf_digits and
// k_pf_digits_long (hx_prefill.cu) share.
//
// A value becomes the integer X = round(x / S_b * 2^27), |X| <= 2^28, spelled with eight base-13 digits.  S_b is the power of two at or below
// the largest element of the value's block, at least 2^-9 S (S: the same of the whole vector).  A block is what a byte of column scales
// stands for: 16 columns of K in an MMA step of 64, and with the same bytes used for two steps the 16 at the same place of the next step: 32
// columns (128 h + 16 j + i and 128 h + 64 + 16 j + i, i < 16).  What a large element costs is the resolution of the 31 values beside it.  (One
// scale per 256 columns: rows whose weight on the large element is zero had up to 2.9 times the error.  A scale per 16 columns takes
// twice the shared memory and a slot of the ring of weight cells at 26 tokens.)
//
// The digit values 0, 1, 2, 3, 4, 6, 8 and their negatives
// are E2M1 values (times two) and one of each residue modulo 13 (5 = -8, 7 = -6); eight of them spell every integer below
// 5 * 13^7 - 8 (13^7 - 1) / 12 = 2^28.02.  Two digits at a time: X modulo 169 is an index into a table of bytes with the two E2M1
// codes, whose top bit -- the sign of the pair, a negative zero where only the lower digit is negative -- is what the quotient is
// carried up by.
#pragma once
#include "hx_gemm_tc.cuh"

#define HX_DIG_CODES 169
// table entry `i`: residue -> the codes of two digits, the more significant one in the high nibble
__device__ __forceinline__ uint8_t dig_code(int i) {
    constexpr unsigned long long NIB = 0x9ABC6D5E43210ull;      // codes of the residues 0 .. 12: 0 1 2 3 4 -8 6 -6 8 -4 -3 -2 -1
    const uint32_t h = (uint32_t)i / 13u, l = (uint32_t)i - 13u * h, lo = (uint32_t)(NIB >> (4 * l)) & 0xFu, h1 = h + (lo >> 3);
    return (uint8_t)((h1 < 13u ? ((uint32_t)(NIB >> (4 * h1)) & 0xFu) << 4 : 0x80u) | lo);
}
// the power of two at or below a vector's largest element (1 for zero and for what is not finite)
__device__ __forceinline__ float dig_scale(float vmax) {
    return vmax > 0.0f && vmax < INFINITY ? __uint_as_float(__float_as_uint(vmax) & 0x7F800000u) : 1.0f;
}
// the largest of eight consecutive values of each lane's block (lane: columns 8 lane .. 8 lane + 7 of a cell of 256)
__device__ __forceinline__ float dig_block_max(const float (&v)[8]) {
    float m = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; e++) m = fmaxf(m, fabsf(v[e]));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    return fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
}
// r with S_b = 2^-r S for a block whose largest element is bm: 0 .. 9, the range of an E4M3 scale (r stops where 2^27 / S_b would overflow)
__device__ __forceinline__ int dig_block_exp(float S, float bm) {
    return min(9, max(0, (int)(__float_as_uint(S) >> 23) - max(40, (int)(__float_as_uint(bm) >> 23))));
}
// E4M3 of 2^-r (2^-7 and below are subnormal)
__device__ __forceinline__ uint32_t dig_block_sf(int r) { return r < 7 ? (uint32_t)(7 - r) << 3 : 4u >> (r - 7); }
// eight consecutive values -> one word of eight codes per digit, the most significant digit first
__device__ __forceinline__ void dig_words(const float (&v)[8], float mul, const uint8_t* codes, uint32_t (&word)[HX_TC_DIGITS]) {
    // four pairs (base 169) per element, each a byte of two codes; the bytes of the even and of the odd elements are collected in
    // a word each
    uint32_t ev[HX_TC_DIGITS / 2], od[HX_TC_DIGITS / 2];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        uint32_t q = 815730721u + (uint32_t)__float2int_rn(v[e] * mul);             // 13^8 + X
#pragma unroll
        for (int i = HX_TC_DIGITS / 2 - 1; i >= 0; i--) {
            // q / 169; after the first step q is below 2^32 / 169 and ceil(2^32 / 169) needs no shift
            const uint32_t qn = i == HX_TC_DIGITS / 2 - 1 ? q / 169u : __umulhi(q, 25414008u), c = codes[q - qn * 169u];
            uint32_t& to = (e & 1) ? od[i] : ev[i];
            to = e < 2 ? c : to + (c << (8 * (e >> 1)));
            q = qn + (c >> 7);
        }
        if (e & 1) asm volatile("" ::: "memory");        // two elements at a time: fewer registers
    }
#pragma unroll
    for (int i = 0; i < HX_TC_DIGITS / 2; i++) {
        word[2 * i] = ((ev[i] >> 4) & 0x0F0F0F0Fu) | (od[i] & 0xF0F0F0F0u);         // the more significant digit of the pair
        word[2 * i + 1] = (ev[i] & 0x0F0F0F0Fu) | ((od[i] << 4) & 0xF0F0F0F0u);
    }
}
// The words of a warp's lanes (lane: columns 8 lane .. 8 lane + 7 of the cell) to token tl's rows of a cell, and the column scales of its blocks.
// Tokens go in pairs: digit d of token tl is row 16 (tl / 2) + 2 d + tl % 2, so that the read-out finds the same digit of two tokens side
// by side.  Rows are 128 bytes, 16-byte chunk j at place j ^ (row % 8); the scales lie as tcgen05.cp wants them.
__device__ __forceinline__ void dig_store(uint8_t* cell, int group, int tl, int lane, const uint32_t (&word)[HX_TC_DIGITS], int r) {
    uint8_t* dst = cell + (tl >> 1) * 2048 + (tl & 1) * 128 + (lane & 3) * 4;
    const int j = (lane >> 2) ^ (tl & 1);
#pragma unroll
    for (int n = 0; n < HX_TC_DIGITS; n++) *reinterpret_cast<uint32_t*>(dst + n * 256 + ((j ^ ((2 * n) & 7)) << 4)) = word[n];
    uint32_t sf = dig_block_sf(r) << (8 * ((lane >> 1) & 3));        // byte j: block j of the lane's half of the cell
    sf |= __shfl_xor_sync(0xffffffffu, sf, 2);
    sf |= __shfl_xor_sync(0xffffffffu, sf, 4);
    if ((lane & 8) == 0) {
        const uint32_t row = (uint32_t)((tl >> 1) * 16 + (lane & 7) * 2 + (tl & 1));
        *reinterpret_cast<uint32_t*>(cell + group * 1024 + (lane >> 4) * HX_TC_DSF(group) + (row >> 7) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4) = sf;
    }
}
