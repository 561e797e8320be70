// Pieces of the head_dim-256 decode bodies that read q8_0 / q4_0 rows as they lie in the cache:
// the order in which a lane takes code bytes out of a row, their conversion to f16 operands and the
// f16 MMA.
#pragma once

#include "params.cuh"
#include "q8_pack.cuh"

namespace hipml {

constexpr int kTile = 64;                        // rows per unit of the run plan
constexpr int kRowBytes = 8 * kQ8BlockBytes;     // 272
constexpr int kQ4RowBytes = 8 * kQ4BlockBytes;   // 144 = 36 words; a block pair is 9 words
constexpr float kPScale = 1024.0f;               // keeps weight*scale in f16's normal range
constexpr float kPScaleLog2 = 10.0f;
constexpr unsigned kSpinLimit = 1u << 24;        // polls of a full barrier before giving up

// d = a * b + c (a, b f16; c, d f32)
__device__ __forceinline__ void mma_16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1,
                                          const float (&c)[4]) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%10,%11,%12,%13};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]),
          "f"(c[3]));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    mma_16816(c, a, b0, b1, c);
}

// The code bytes of a q8_0 block as eight "logical words" (four codes each), all 4-byte aligned. Odd
// blocks start 2 bytes past a word boundary, so word j holds codes 4j..4j+3. Even blocks start on a
// word boundary (the scale shares a word with codes 0, 1): words 0..6 hold codes 4j+2..4j+5 and word 7
// is stitched from codes 0, 1 and 30, 31. The order of elements inside the contraction is free as
// long as the query operand uses the same one. This is the head_dim index of byte i of word j.
__device__ __forceinline__ int k_word_dim(int blk, int j, int i) {
    if (blk & 1) return blk * 32 + 4 * j + i;
    if (j < 7) return blk * 32 + 4 * j + 2 + i;
    return blk * 32 + (i < 2 ? i : 28 + i);
}

// Two bytes of `biased` (code ^ 0x80 = code + 128) as a half2 of f16 subnormals: 0x00xx is
// xx * 2^-24 exactly, so one permute converts two codes. The offset of 128 is taken out
// again through the accumulators, the factor 2^-24 when the scores are read.
__device__ __forceinline__ unsigned codes_to_half2(unsigned biased, unsigned selector) {
    return __byte_perm(biased, 0u, selector);
}
constexpr float kCodeUnit = 16777216.0f;          // 2^24
constexpr float kCodeBias = 128.0f / 16777216.0f; // the offset in the operand's units: 2^-17

// The same for a q4_0 block's four words of code bytes (low nibble; the high nibble is 16 further).
__device__ __forceinline__ int k_word_dim_q4(int blk, int j, int i) {
    if (blk & 1) return blk * 32 + 4 * j + i;
    if (j < 3) return blk * 32 + 4 * j + 2 + i;
    return blk * 32 + (i < 2 ? i : 12 + i);
}

}  // namespace hipml
