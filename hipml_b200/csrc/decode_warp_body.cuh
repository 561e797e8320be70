// The pieces of the decode body whose warps work alone (attn_decode_warps.cu) that its form for several
// columns of one stream (attn_decode_cols.cu) shares, operation for operation: a column's result does
// not depend on which of the two computed it.
#pragma once

#include <type_traits>

#include "decode_fold.cuh"
#include "decode_rows.cuh"
#include "params.cuh"
#include "sm100_ptx.cuh"

namespace hipml {
namespace warp_body {

using namespace ptx;

template <int N>
using Int = std::integral_constant<int, N>;

constexpr int kWarps = 8;                        // per CTA
constexpr int kThreads = 32 * kWarps;
constexpr int kHeadPitch = 260;                  // floats per head of a warp's partial (bank spread)
// A reference is set this far (log2) above the maximum seen, so that the few units a warp takes
// rarely move it again: with the exact maximum 75 % of the units of a 100,000-row step rescaled 64
// accumulators.
constexpr float kMargin = 1.5f;
constexpr int kNeutralSlots = 32;   // partial slots that are written whether or not a run of rows has them
constexpr int kPrefetch = 2;   // units of K and of V a warp asks L2 for ahead of the grid dependency

// Transpose of an 8 x 8 tile of f16 held one 32-bit pair per lane (row = lane / 4).
__device__ __forceinline__ unsigned transpose8(unsigned x) {
    unsigned y;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
__device__ __forceinline__ void split2(float a, float b, unsigned &hi, unsigned &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const unsigned *>(&h);
    lo = *reinterpret_cast<const unsigned *>(&l);
}

// A pair of blocks (2M, 2M + 1) of a row is a whole number of words from a word boundary: W[0] =
// {scale of the even block, its codes 0, 1}, W[kHalf] = {its last two code bytes, scale of the odd
// block}, then the odd block's code words. So every code word but one is an aligned word of the
// row: the even block's word j holds code bytes 4j + 2 .. 4j + 5, and its last one is stitched from
// the outer two words, whose other halves are the scales.
template <bool kQ4>
struct Row {
    static constexpr int kWords = kQ4 ? 4 : 8;         // code words of a block
    static constexpr int kHalf = kWords;               // the word with the odd block's scale
    static constexpr int kPair = 2 * kWords + 1;       // words of a pair
    static constexpr int kPitch = kQ4 ? kQ4RowBytes / 4 : kRowBytes / 4;
};
__device__ __forceinline__ unsigned stitch(unsigned w0, unsigned wh) { return __byte_perm(w0, wh, 0x5432); }
__device__ __forceinline__ float low_half(unsigned w) { return half_bits_to_float((unsigned short)w); }
__device__ __forceinline__ float high_half(unsigned w) { return half_bits_to_float((unsigned short)(w >> 16)); }

// Query fragments of one block (the warp's) into `frag`: for each of its two 16-slot steps the B
// operand's {hi b0, hi b1, lo b0, lo b1} of column g (head g; heads past the group are zero), slots in the
// order of k_word_dim (2t, 2t + 1 = bytes 0, 1 of word t; 2t + 8, 2t + 9 = bytes 2, 3); x holds the lane's values
// in that order. And the C operand that takes the codes' offset of 128 (nibbles: 8) out: -2^-17 * their
// sum, as {head 2t, 2t + 1, 2t, 2t + 1}.
template <bool kQ4>
__device__ __forceinline__ void store_query(const float2 (&x)[2][2], float scale_log2, int blk, int lane, uint4 *frag,
                                            float *bias) {
    const int g = lane >> 2, t = lane & 3;
    float sum = 0.0f;   // of the block's query values as the tensor cores see them
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint4 f;
        split2(x[k][0].x * scale_log2, x[k][0].y * scale_log2, f.x, f.z);
        split2(x[k][1].x * scale_log2, x[k][1].y * scale_log2, f.y, f.w);
        const unsigned v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 y = __half22float2(*reinterpret_cast<const __half2 *>(&v[i]));
            sum += y.x + y.y;
        }
        frag[(2 * blk + k) * 32 + lane] = f;
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (t == 0) {
        float *const dst = bias + blk * 16 + (g >> 1) * 4 + (g & 1);
        dst[0] = dst[2] = -(kQ4 ? kCodeBias / 16.0f : kCodeBias) * sum;
    }
}

// ---- scores. A warp's K operands of blocks 2M, 2M + 1 for kT tiles of 16 rows.
template <int kT>
struct KFrag {
    unsigned e[2][kT][4], o[2][kT][4];   // [16-slot step][tile]: A fragment of the even / odd block
    float de[kT][2], dd[kT][2];          // their scales, rows g and g + 8
};
template <int M, bool kQ4, int kT>
__device__ __forceinline__ void load_k(const unsigned *row, int t, KFrag<kT> &f) {
    using R = Row<kQ4>;
#pragma unroll
    for (int i = 0; i < kT; i++) {
        unsigned e[2][2], o[2][2];       // [step][row g, g + 8]: biased codes
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const unsigned *w = row + (i * 16 + r * 8) * R::kPitch + M * R::kPair;
            const unsigned w0 = w[0], wh = w[R::kHalf];
            f.de[i][r] = low_half(w0);
            f.dd[i][r] = high_half(wh);
            if constexpr (kQ4) {
                const unsigned x = w[1 + t], y = w[5 + t];
                const unsigned ev = t == 3 ? stitch(w0, wh) : x;
                e[0][r] = ev & 0x0f0f0f0fu;
                e[1][r] = (ev >> 4) & 0x0f0f0f0fu;
                o[0][r] = y & 0x0f0f0f0fu;
                o[1][r] = (y >> 4) & 0x0f0f0f0fu;
            } else {
                const unsigned x0 = w[1 + t], x1 = w[5 + t];
                e[0][r] = x0 ^ 0x80808080u;
                e[1][r] = (t == 3 ? stitch(w0, wh) : x1) ^ 0x80808080u;
                o[0][r] = w[9 + t] ^ 0x80808080u;
                o[1][r] = w[13 + t] ^ 0x80808080u;
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                f.e[k][i][c] = codes_to_half2(e[k][c & 1], c < 2 ? 0x4140 : 0x4342);
                f.o[k][i][c] = codes_to_half2(o[k][c & 1], c < 2 ? 0x4140 : 0x4342);
            }
    }
}
// Adds the two blocks' scores into s: s[i][0], s[i][1] = row g of tile i, heads 2t and 2t + 1; s[i][2],
// s[i][3] = row g + 8. A query fragment serves all tiles; the MMA chains of tiles and blocks interleave.
template <int M, int kT>
__device__ __forceinline__ void add_scores(const KFrag<kT> &f, const uint4 *qf, const float4 *bias, float (&s)[kT][4]) {
    const float4 be = bias[2 * M * 4], bo = bias[(2 * M + 1) * 4];
    const float c0e[4] = {be.x, be.y, be.z, be.w}, c0o[4] = {bo.x, bo.y, bo.z, bo.w};
    float ce[kT][4], co[kT][4];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint4 qe = qf[(4 * M + k) * 32], qo = qf[(4 * M + 2 + k) * 32];
#pragma unroll
        for (int i = 0; i < kT; i++) {
            if (k == 0) {
                mma_16816(ce[i], f.e[k][i], qe.x, qe.y, c0e);
                mma_16816(co[i], f.o[k][i], qo.x, qo.y, c0o);
            } else {
                mma_16816(ce[i], f.e[k][i], qe.x, qe.y);
                mma_16816(co[i], f.o[k][i], qo.x, qo.y);
            }
        }
#pragma unroll
        for (int i = 0; i < kT; i++) {
            mma_16816(ce[i], f.e[k][i], qe.z, qe.w);
            mma_16816(co[i], f.o[k][i], qo.z, qo.w);
        }
    }
#pragma unroll
    for (int i = 0; i < kT; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) s[i][c] = fmaf(f.dd[i][c >> 1], co[i][c], fmaf(f.de[i][c >> 1], ce[i][c], s[i][c]));
}

// ---- softmax of a unit: running reference and sum of a lane's heads 2t, 2t + 1.
struct Running {
    float m[2], nm[2], l[2];   // reference, 10 - reference, sum (of this lane's rows)
};
__device__ __forceinline__ void start(Running &r) {
    r.m[0] = r.m[1] = -INFINITY;
    r.nm[0] = r.nm[1] = INFINITY;
    r.l[0] = r.l[1] = 0.0f;
}
__device__ __forceinline__ void sum_rows(Running &r) {   // over the lanes of a head
#pragma unroll
    for (int h = 0; h < 2; h++) {
        r.l[h] += __shfl_xor_sync(0xffffffffu, r.l[h], 4);
        r.l[h] += __shfl_xor_sync(0xffffffffu, r.l[h], 8);
        r.l[h] += __shfl_xor_sync(0xffffffffu, r.l[h], 16);
    }
}
// The exponents score - reference + 10 of kT tiles. Rows from rows[h] on are out of head 2t + h's sight; with kApart the
// heads differ in that, and one may see none (rows[h] <= 0). over[h]: one of the lane's scores is above the head's
// reference (not kApart: over[0], of either head).
template <int kT, bool kApart>
__device__ __forceinline__ void exponents(float (&s)[kT][4], const int (&rows)[2], int g, const Running &r, float (&nm)[2],
                                          float (&x)[kT][4], bool (&over)[2]) {
    nm[0] = r.nm[0];
    nm[1] = r.nm[1];
    if ((kApart ? min(rows[0], rows[1]) : rows[0]) < 16 * kT) {   // rows past the end hold stale bytes
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (kApart && rows[h] <= 0) nm[h] = 0.0f;   // (-infinity from here on, not NaN)
#pragma unroll
            for (int j = 0; j < kT; j++) {
                if (16 * j + g >= rows[kApart ? h : 0]) s[j][h] = -INFINITY;
                if (16 * j + g + 8 >= rows[kApart ? h : 0]) s[j][h + 2] = -INFINITY;
            }
        }
    }
    float xm[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < kT; j++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            x[j][c] = fmaf(s[j][c], kCodeUnit, nm[c & 1]);
            float &m = xm[kApart ? c & 1 : 0];
            m = fmaxf(m, x[j][c]);
        }
    over[0] = xm[0] > kPScaleLog2;
    over[1] = xm[1] > kPScaleLog2;
}
// Moving the references of one column's heads: all of them as soon as one is exceeded.
struct MoveAll {
    __device__ __forceinline__ bool operator()(const bool (&over)[2], bool (&move)[2]) const {
        return move[0] = move[1] = __any_sync(0xffffffffu, over[0] || over[1]);
    }
};
// The weights 2^(score - reference + 10) of kT tiles, as f16 high and low pairs in the B operand's
// layout: ph[j][0] = rows 2t, 2t + 1 of tile j for head g, ph[j][1] = rows 2t + 8, 2t + 9; weight 0 out of sight, and a
// head that sees no row keeps its state. True when references moved: what was accumulated must be multiplied by corr.
template <int kT, bool kApart = false, class Move = MoveAll>
__device__ __forceinline__ bool softmax(float (&s)[kT][4], const int (&rows)[2], int g, Running &r, __half2 (&ph)[kT][2],
                                        __half2 (&pl)[kT][2], float (&corr)[2], Move decide = {}) {
    float nm[2], x[kT][4];
    bool over[2], move[2];
    exponents<kT, kApart>(s, rows, g, r, nm, x, over);
    const bool moved = decide(over, move);
    if (moved) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < kT; j++) mx = fmaxf(mx, fmaxf(s[j][h], s[j][h + 2]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            // (rounded up to 1/16, so that the shift by 10 is exact)
            const float top = ceilf(mx * (kCodeUnit * 16.0f)) * 0.0625f;
            const float mn = top > r.m[h] ? top + kMargin : r.m[h];
            corr[h] = 1.0f;
            if (!kApart || (move[h] && rows[h] > 0)) {
                corr[h] = ex2(r.m[h] - mn);
                r.m[h] = mn;
                r.nm[h] = nm[h] = kPScaleLog2 - mn;
                r.l[h] *= corr[h];
            }
        }
#pragma unroll
        for (int j = 0; j < kT; j++)
#pragma unroll
            for (int c = 0; c < 4; c++) x[j][c] = fmaf(s[j][c], kCodeUnit, nm[c & 1]);
    }
#pragma unroll
    for (int j = 0; j < kT; j++) {
        float pw[4];
#pragma unroll
        for (int c = 0; c < 4; c++) pw[c] = ex2(x[j][c]);
        r.l[0] += pw[0] + pw[2];
        r.l[1] += pw[1] + pw[3];
#pragma unroll
        for (int c = 0; c < 2; c++) {
            unsigned hi, lo;
            split2(pw[2 * c], pw[2 * c + 1], hi, lo);
            hi = transpose8(hi);
            lo = transpose8(lo);
            ph[j][c] = *reinterpret_cast<const __half2 *>(&hi);
            pl[j][c] = *reinterpret_cast<const __half2 *>(&lo);
        }
    }
    return moved;
}

// ---- values. A warp's V operands of blocks 2M, 2M + 1 for one tile of 16 rows (`row`: its row 2t).
struct VFrag {
    unsigned e[2][4], o[2][4];         // A fragments of the even / odd block: two code bytes of the lane's of each row (see value_dim)
    __half2 de01, de23, do01, do23;    // scales of rows 2t, 2t + 1 / 2t + 8, 2t + 9
};
__device__ __forceinline__ __half2 as_half2(unsigned x) { return *reinterpret_cast<const __half2 *>(&x); }
__device__ __forceinline__ unsigned as_bits(const __half2 &x) { return *reinterpret_cast<const unsigned *>(&x); }
// q8_0: code bytes {0, 1} and {2, 3} of word g of each row.
template <int M>
__device__ __forceinline__ void load_v_q8(const unsigned *row, int g, VFrag &f) {
    using R = Row<false>;
    constexpr int kRowOf[4] = {0, 1, 8, 9};
    unsigned w0[4], wh[4], we[4], wo[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const unsigned *w = row + kRowOf[e] * R::kPitch + M * R::kPair;
        w0[e] = w[0];
        wh[e] = w[R::kHalf];
        we[e] = w[1 + g];
        wo[e] = w[R::kHalf + 1 + g];
    }
    auto convert = [&](unsigned (&x)[4], unsigned (&a)[2][4]) {
#pragma unroll
        for (int e = 0; e < 4; e++) x[e] ^= 0x80808080u;
        // 0x64xx = 1024 + xx, minus 1152: exact. (The weights are all positive, an offset
        // left to the accumulators would cost several bits: 4e-5 relative on a flat 256-key run.)
        auto conv = [&](unsigned y, unsigned sel) {
            return as_bits(__hsub2(as_half2(__byte_perm(y, 0x64646464u, sel)), as_half2(0x64806480u)));
        };
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const unsigned ab = __byte_perm(x[0], x[1], i ? 0x7362 : 0x5140);   // [a0 b0 a1 b1] / [a2 b2 a3 b3]
            const unsigned cd = __byte_perm(x[2], x[3], i ? 0x7362 : 0x5140);
            a[i][0] = conv(ab, 0x4140);
            a[i][1] = conv(ab, 0x4342);
            a[i][2] = conv(cd, 0x4140);
            a[i][3] = conv(cd, 0x4342);
        }
    };
#pragma unroll
    for (int e = 0; e < 4; e++) we[e] = g == R::kWords - 1 ? stitch(w0[e], wh[e]) : we[e];
    f.de01 = as_half2(__byte_perm(w0[0], w0[1], 0x5410));
    f.de23 = as_half2(__byte_perm(w0[2], w0[3], 0x5410));
    f.do01 = as_half2(__byte_perm(wh[0], wh[1], 0x7632));
    f.do23 = as_half2(__byte_perm(wh[2], wh[3], 0x7632));
    convert(we, f.e);
    convert(wo, f.o);
}
// q4_0: the low (i = 0) and the high nibbles of code bytes 2g and 2g + 1 of each row. Both nibbles of a byte serve the
// same lane, and its two bytes are a half word, so that a pair of rows is one word and a nibble of it one mask: ten
// instructions for eight values and none to stitch a word across the scale, where a word a row with one nibble of each
// byte took 14 and four more (30,000 rows: 19.2 -> 18.8 us a layer; two slots of up to 6,667: 13.5 -> 13.3).
template <int M>
__device__ __forceinline__ void load_v_q4(const unsigned *row, int g, VFrag &f) {
    using R = Row<true>;
    constexpr int kRowOf[4] = {0, 1, 8, 9};
    unsigned se[4], so[4], ce[4], co[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const unsigned short *w = reinterpret_cast<const unsigned short *>(row + kRowOf[e] * R::kPitch + M * R::kPair);
        se[e] = w[0];
        ce[e] = w[1 + g];
        so[e] = w[R::kPair];
        co[e] = w[R::kPair + 1 + g];
    }
    auto both = [](unsigned lo, unsigned hi) { return __byte_perm(lo, hi, 0x5410); };
    auto convert = [&](const unsigned (&x)[4], unsigned (&a)[2][4]) {
#pragma unroll
        for (int p = 0; p < 2; p++) {   // rows 2t, 2t + 1 / 2t + 8, 2t + 9
            const unsigned y = both(x[2 * p], x[2 * p + 1]);
#pragma unroll
            for (int byte = 0; byte < 2; byte++) {
                const unsigned z = y >> (8 * byte);
                // 1024 + n, minus 1032; (1024 + 16 n) / 16 - 72: both exact
                a[0][2 * p + byte] = as_bits(__hsub2(as_half2((z & 0x000f000fu) | 0x64006400u), as_half2(0x64086408u)));
                a[1][2 * p + byte] = as_bits(__hfma2(as_half2((z & 0x00f000f0u) | 0x64006400u), as_half2(0x2c002c00u),
                                                     as_half2(0xd480d480u)));
            }
        }
    };
    f.de01 = as_half2(both(se[0], se[1]));
    f.de23 = as_half2(both(se[2], se[3]));
    f.do01 = as_half2(both(so[0], so[1]));
    f.do23 = as_half2(both(so[2], so[3]));
    convert(ce, f.e);
    convert(co, f.o);
}
template <int M, bool kQ4>
__device__ __forceinline__ void load_v(const unsigned *row, int g, VFrag &f) {
    if constexpr (kQ4)
        load_v_q4<M>(row, g, f);
    else
        load_v_q8<M>(row, g, f);
}
// acc[block][i][c] += weights * values, c = {dim, dim + 1} x {head 2t, 2t + 1} from value_dim(block, g, i) on.
// kMasked: heads g of lanes without `keep` get nothing, whatever the rows' scales are.
template <bool kMasked = false>
__device__ __forceinline__ void add_values(const VFrag &f, const __half2 (&ph)[2], const __half2 (&pl)[2],
                                           float (&acc_e)[2][4], float (&acc_o)[2][4], bool keep = true) {
    auto bits = [&](const __half2 &h) { return !kMasked || keep ? *reinterpret_cast<const unsigned *>(&h) : 0u; };
    auto block = [&](const __half2 d01, const __half2 d23, const unsigned (&a)[2][4], float (&acc)[2][4]) {
        const __half2 h01 = __hmul2(ph[0], d01), h23 = __hmul2(ph[1], d23);
        const __half2 l01 = __hfma2(pl[0], d01, __hfma2(ph[0], d01, __hneg2(h01)));
        const __half2 l23 = __hfma2(pl[1], d23, __hfma2(ph[1], d23, __hneg2(h23)));
#pragma unroll
        for (int i = 0; i < 2; i++) {
            mma_16816(acc[i], a[i], bits(h01), bits(h23));
            mma_16816(acc[i], a[i], bits(l01), bits(l23));
        }
    };
    block(f.de01, f.de23, f.e, acc_e);
    block(f.do01, f.do23, f.o, acc_o);
}
// First of the two dims (within the block) that lane group g has in half 0 and in half 1 of its operands: q8_0 code bytes
// {0, 1} and {2, 3} of its word (of an even block, whose words begin with byte 2, the last is stitched); q4_0 the low and
// the high nibbles of its two bytes.
template <bool kQ4>
__device__ __forceinline__ int value_dim(int blk, int g, int half) {
    if (kQ4) return 2 * g + 16 * half;
    if (blk & 1) return 4 * g + 2 * half;
    if (g == Row<false>::kWords - 1) return half ? 30 : 0;
    return 4 * g + 2 + 2 * half;
}

// Whether the CTA that folds slice `rank` of the items writes the {maximum, sum} of this item's head to memory: with
// the first item of the head, and with the first of the slice where that lies inside a head. The counter of the runs is
// one per slice, so whoever folds the slice there may only read what CTAs of the same rank wrote; the CTAs that share a
// head write the same bits.
template <int kC>
__device__ __forceinline__ bool writes_pair(int items, int rank, int item) {
    return (item & 63) == 0 || item == items * rank / kC;
}

// ---- folds. A partial of a head is (acc, m, l) with weights relative to 2^m and 2^10 too large, as the warps add them
// up; the scale leaves where a sum is divided by another, or with the row of a shard. (Left out of every warp's m instead,
// ahead of the first fold, it cost 0.5 us of the 99 that 16 layers of 672 rows take.) Folding partials is associative up
// to rounding, and always runs in one order with explicit operations.
struct Part {
    float4 a;
    float m, l;
};
__device__ __forceinline__ void rescale(Part &r, float big) {
    const float c = r.m == -INFINITY ? 0.0f : ex2(r.m - big);
    r.a.x = __fmul_rn(r.a.x, c);
    r.a.y = __fmul_rn(r.a.y, c);
    r.a.z = __fmul_rn(r.a.z, c);
    r.a.w = __fmul_rn(r.a.w, c);
    r.l = __fmul_rn(r.l, c);
    r.m = big;
}
__device__ __forceinline__ void add(Part &r, const float4 &x, const float2 &ml) {   // r.m >= ml.x
    const float w = ml.x == -INFINITY ? 0.0f : ex2(ml.x - r.m);
    r.a.x = fmaf(x.x, w, r.a.x);
    r.a.y = fmaf(x.y, w, r.a.y);
    r.a.z = fmaf(x.z, w, r.a.z);
    r.a.w = fmaf(x.w, w, r.a.w);
    r.l = fmaf(ml.y, w, r.l);
}

// Folds sources [i0, i1) of kPer items each: load(i, j, x, ml) fetches source i of item j. The loads of
// kBatch sources are issued together: a batch costs one round trip.
template <int kPer, int kBatch, class Load>
__device__ __forceinline__ void fold_sources(int i0, int i1, Load load, Part (&r)[kPer]) {
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        r[j].a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        r[j].m = -INFINITY;
        r[j].l = 0.0f;
    }
    for (int s0 = i0; s0 < i1; s0 += kBatch) {
        float4 x[kPer][kBatch];
        float2 ml[kPer][kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; i++)
#pragma unroll
            for (int j = 0; j < kPer; j++) {
                x[j][i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                ml[j][i] = make_float2(-INFINITY, 0.0f);
                if (s0 + i < i1) load(s0 + i, j, x[j][i], ml[j][i]);
            }
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            float big = r[j].m;
#pragma unroll
            for (int i = 0; i < kBatch; i++) big = fmaxf(big, ml[j][i].x);
            rescale(r[j], big);
#pragma unroll
            for (int i = 0; i < kBatch; i++) add(r[j], x[j][i], ml[j][i]);
        }
    }
}

// The same for the sources of one item in memory, independent of the batch: the maximum first (from the {m, l} pairs
// alone where there is more than one batch), then the sum in source order.
template <int kBatch, class LoadMl, class Load>
__device__ __forceinline__ void fold_memory(int i0, int i1, LoadMl load_ml, Load load, Part &r) {
    r.a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    r.m = -INFINITY;
    r.l = 0.0f;
    const bool one_batch = i1 - i0 <= kBatch;
    if (!one_batch) {
        for (int s0 = i0; s0 < i1; s0 += 16)
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (s0 + i < i1) r.m = fmaxf(r.m, load_ml(s0 + i).x);
    }
    for (int s0 = i0; s0 < i1; s0 += kBatch) {
        float4 x[kBatch];
        float2 ml[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
            x[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            ml[i] = make_float2(-INFINITY, 0.0f);
            if (s0 + i < i1) {
                x[i] = load(s0 + i);
                ml[i] = load_ml(s0 + i);
            }
        }
        if (one_batch)
#pragma unroll
            for (int i = 0; i < kBatch; i++) r.m = fmaxf(r.m, ml[i].x);
#pragma unroll
        for (int i = 0; i < kBatch; i++) add(r, x[i], ml[i]);
    }
}

// In a cluster of kC a CTA has 1 / kC of a head group's items (at most 512) to fold: kShare neighbouring
// threads take an item, each with a contiguous share of the sources, joined by shuffles.
template <int kC>
struct Split {
    static constexpr int kShare = kC > 2 ? kC / 2 : 1;
};
template <int kShare>
__device__ __forceinline__ void join(Part &r) {
#pragma unroll
    for (int o = 1; o < kShare; o <<= 1) {
        float4 x;
        float2 ml;
        x.x = __shfl_xor_sync(0xffffffffu, r.a.x, o);
        x.y = __shfl_xor_sync(0xffffffffu, r.a.y, o);
        x.z = __shfl_xor_sync(0xffffffffu, r.a.z, o);
        x.w = __shfl_xor_sync(0xffffffffu, r.a.w, o);
        ml.x = __shfl_xor_sync(0xffffffffu, r.m, o);
        ml.y = __shfl_xor_sync(0xffffffffu, r.l, o);
        rescale(r, fmaxf(r.m, ml.x));
        add(r, x, ml);
    }
}

// A warp's accumulators as a partial [head][dims] with kHeadPitch floats per head.
template <bool kQ4>
__device__ __forceinline__ void store_warp_partial(float *dst, const float (&acc)[8][2][4], int group, int g, int t) {
#pragma unroll
    for (int h = 0; h < 2; h++)
        if (2 * t + h < group) {
#pragma unroll
            for (int b = 0; b < 8; b++)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    *reinterpret_cast<float2 *>(dst + (2 * t + h) * kHeadPitch + 32 * b + value_dim<kQ4>(b, g, i)) =
                        make_float2(acc[b][i][h], acc[b][i][2 + h]);
        }
}
// Folds the partials of a CTA's warps (`pitch` bytes apart; ml: [8 heads][warp]); done(item, part).
template <class Done>
__device__ __forceinline__ void fold_warps(const unsigned char *partials, int pitch, const float2 *ml_at, int items,
                                           Done done) {
    constexpr int kPer = 2;   // (at most 512 items)
    const int tid = threadIdx.x;
    Part r[kPer];
    fold_sources<kPer, kWarps>(
        0, kWarps,
        [&](int i, int j, float4 &x, float2 &ml) {
            const int item = min(tid + j * kThreads, items - 1);
            x = *reinterpret_cast<const float4 *>(partials + i * pitch + ((item >> 6) * kHeadPitch + 4 * (item & 63)) * 4);
            ml = ml_at[(item >> 6) * kWarps + i];
        },
        r);
#pragma unroll
    for (int j = 0; j < kPer; j++)
        if (tid + j * kThreads < items) done(tid + j * kThreads, r[j]);
}
// Merge of a cluster by reading: folds slice `rank` of the items of the kC CTAs of a cluster (partials of [item] at
// cpart, {max, sum} of [8 heads] at cml, at the same place in each CTA), for threads 0 .. kThreads - 1 or more;
// done(item, part).
template <int kC, class Done>
__device__ __forceinline__ void fold_cluster(const float4 *cpart, const float2 *cml, int items, int rank, Done done) {
    constexpr int kShare = Split<kC>::kShare;
    static_assert(kC % kShare == 0 && 512 / kC * kShare <= kThreads, "slices");
    const int first = items * rank / kC, count = items * (rank + 1) / kC - first;
    const int at = threadIdx.x / kShare, part = threadIdx.x % kShare, item = first + min(at, count - 1);
    if ((int)(threadIdx.x & ~31u) / kShare >= count) return;   // (whole warps: the others join by shuffles)
    Part r[1];
    fold_sources<1, kC / kShare>(
        part * (kC / kShare), (part + 1) * (kC / kShare),
        [&](int i, int, float4 &x, float2 &ml) {
            x = ld_cluster_f4(map_to_cta(smem_u32(cpart + item), i));
            ml = ld_cluster_f2(map_to_cta(smem_u32(cml + (item >> 6)), i));
        },
        r);
    join<kShare>(r[0]);
    if (at < count && part == 0) done(item, r[0]);
}

// Merge of a cluster, one column: every CTA sends each item of its partial to the CTA that folds it (slice r of
// the items: CTA r) as soon as it has it, and that one waits on its own barrier and reads locally; none has to
// stay for another's reads. (A barrier of the cluster, remote loads and another barrier were 0.9 us of the 8.3 us
// that a layer of 672 rows took, 0.7 of 14.9 with its front end at 8,192 rows, 0.6 of 12.6 over the f32 cache at
// 2,048. Several columns, whose partials would need an inbox each, are read: fold_cluster.)
// inbox: [kC sources][items / kC] float4, inbox_ml: [kC][8 heads]; kC divides 64. The receiver's barrier expects
// inbox_bytes.
template <int kC>
__device__ __forceinline__ unsigned inbox_bytes(int items, int rank) {
    const int count = items / kC, first = count * rank;
    const int heads = ((first + count - 1) >> 6) - (first >> 6) + 1;
    return (unsigned)((kC - 1) * (count * 16 + heads * 8));
}
template <int kC>
__device__ __forceinline__ void send_item(float4 *inbox, float2 *inbox_ml, unsigned bar, int items, int rank, int item,
                                          const Part &r) {
    const int count = items / kC, owner = item / count, at = item - owner * count;
    float4 *const to = inbox + rank * count + at;
    float2 *const to_ml = inbox_ml + rank * 8 + (item >> 6);
    const bool with_ml = at == 0 || (item & 63) == 0;   // once per head of the slice
    if (owner == rank) {
        *to = r.a;
        if (with_ml) *to_ml = make_float2(r.m, r.l);
    } else {
        const unsigned remote_bar = map_to_cta(bar, owner);
        st_async_f4(map_to_cta(smem_u32(to), owner), r.a, remote_bar);
        if (with_ml) st_async_f2(map_to_cta(smem_u32(to_ml), owner), make_float2(r.m, r.l), remote_bar);
    }
}
template <int kC, class Done>
__device__ __forceinline__ void fold_inbox(const float4 *inbox, const float2 *inbox_ml, int items, int rank, Done done) {
    constexpr int kShare = Split<kC>::kShare;
    const int count = items / kC, first = count * rank;
    const int at = threadIdx.x / kShare, part = threadIdx.x % kShare, mine = min(at, count - 1), item = first + mine;
    Part r[1];
    fold_sources<1, kC / kShare>(
        part * (kC / kShare), (part + 1) * (kC / kShare),
        [&](int i, int, float4 &x, float2 &ml) {
            x = inbox[i * count + mine];
            ml = inbox_ml[i * 8 + (item >> 6)];
        },
        r);
    join<kShare>(r[0]);
    if (at < count && part == 0) done(item, r[0]);
}
// This CTA's partials of the cluster are all there (its own behind the CTA barrier).
__device__ __forceinline__ bool await_inbox(unsigned bar, unsigned phase) {
    __syncthreads();
    for (unsigned spin = 0; !mbar_try_wait_cluster(bar, phase);)
        if (++spin > kSpinLimit) return false;
    return true;
}

// One float4 (item = head of the group * 64 + dims / 4) of the output: normalised (and gated), or
// the raw triple of a shard, in weights without the scale of 2^10.
__device__ __forceinline__ void emit_item(const DecodeParams &p, int slot, int kvh, int group, int item,
                                          const Part &r) {
    const int h = kvh * group + (item >> 6), j = item & 63;
    const size_t at = (size_t)slot * p.out_slot + (size_t)h * p.out_head_stride + 4 * j;
    float *o = p.out + at;
    if (p.normalize) {
        float4 y;
        y.x = r.l > 0.0f ? __fdiv_rn(r.a.x, r.l) : 0.0f;
        y.y = r.l > 0.0f ? __fdiv_rn(r.a.y, r.l) : 0.0f;
        y.z = r.l > 0.0f ? __fdiv_rn(r.a.z, r.l) : 0.0f;
        y.w = r.l > 0.0f ? __fdiv_rn(r.a.w, r.l) : 0.0f;
        if (p.gate) {
            const float4 g = *reinterpret_cast<const float4 *>(p.gate + at);
            y.x *= 1.0f / (1.0f + expf(-g.x));
            y.y *= 1.0f / (1.0f + expf(-g.y));
            y.z *= 1.0f / (1.0f + expf(-g.z));
            y.w *= 1.0f / (1.0f + expf(-g.w));
        }
        *reinterpret_cast<float4 *>(o) = y;
    } else {
        // rows of head_dim + 2 floats are only 8-byte aligned
        constexpr float kInv = 1.0f / kPScale;
        reinterpret_cast<float2 *>(o)[0] = make_float2(r.a.x * kInv, r.a.y * kInv);
        reinterpret_cast<float2 *>(o)[1] = make_float2(r.a.z * kInv, r.a.w * kInv);
        if (j == 0) {
            o[256] = r.m;
            o[257] = r.l * kInv;
        }
    }
}

// Folds the `runs` partials of slice `rank` of `slices` of a slot's head group from memory and emits it (or, staged !=
// nullptr, leaves it there: [8 heads][256] sums, then [8 heads]{max, sum}). kBatch runs in one round trip: 18 for the
// runs of a deep stream (B200: 18 pairs of SMs per KV head; three trips of 8 took 2.9 us at the end of every launch).
template <int kC, int kBatch>
__device__ __forceinline__ void fold_runs(const DecodeParams &p, int slot, int kvh, int group, int runs, int rank,
                                          float *staged, int slices = kC) {
    constexpr int kShare = Split<kC>::kShare;
    const int items = group * 64, first = items * rank / slices, count = items * (rank + 1) / slices - first;
    const int part = threadIdx.x % kShare, at = threadIdx.x / kShare;
    for (int f0 = at; f0 - at < count; f0 += kThreads / kShare) {   // (whole rounds: the shares join by shuffles)
        const int item = first + min(f0, count - 1), head = kvh * group + (item >> 6);
        const float *const pa = p.part_acc + (size_t)slot * p.acc_slot + (size_t)head * p.splits * 256 + 4 * (item & 63);
        const float *const pm = p.part_ml + (size_t)slot * p.ml_slot + (size_t)head * p.splits * 2;
        Part r;
        fold_memory<kBatch>(
            runs * part / kShare, runs * (part + 1) / kShare,
            [&](int i) { return __ldcg(reinterpret_cast<const float2 *>(pm) + i); },
            [&](int i) { return __ldcg(reinterpret_cast<const float4 *>(pa + (size_t)i * 256)); }, r);
        join<kShare>(r);
        if (f0 >= count || part != 0) continue;
        if (staged) {
            reinterpret_cast<float4 *>(staged)[item] = r.a;
            if ((item & 63) == 0) reinterpret_cast<float2 *>(staged + 8 * 256)[item >> 6] = make_float2(r.m, r.l);
        } else {
            emit_item(p, slot, kvh, group, item, r);
        }
    }
}

// The same fold of all a head group's items, bit for bit, with the partials brought to shared memory by bulk copies: a
// head's runs are one piece of memory, so six heads of 16 runs (98 KB) are six copies. (Ordinary loads keep ~25 KB of a
// CTA's in flight, at ~1 us a trip. Copied run by run, 1 KB each at ~60 ns a copy, they took the last CTA of the head 5
// of the 26 us of a layer of 8 slots of 512 .. 8,192 rows; 16 layers 393 -> 380 us, of 3 slots of up to 3,139 rows 197 ->
// 184.) `area`: `bytes` of shared memory that no copy is in flight to, `bar`: a fresh barrier. False (and nothing done)
// where they do not fit.
constexpr int kStagedRow = 32;   // float2s: {weight, sum} of up to 31 runs, the maximum last
__device__ __forceinline__ bool fold_runs_staged(const DecodeParams &p, int slot, int kvh, int group, int runs,
                                                 unsigned char *area, int bytes, unsigned bar, float2 (*s_ml)[kStagedRow],
                                                 bool &landed) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row = runs * 1024;
    if (runs >= kStagedRow || group * row > bytes) return false;
    // generic writes (of this CTA to the area, of all CTAs to the partials) come before the copies
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, (unsigned)(group * row));
        for (int h = 0; h < group; h++)
            bulk_load(smem_u32(area) + (unsigned)(h * row),
                      p.part_acc + (size_t)slot * p.acc_slot + (size_t)(kvh * group + h) * p.splits * 256, (unsigned)row, bar);
    }
    // weights {2^(m - M), l} of every head, a warp each
    for (int h = warp; h < group; h += kWarps) {
        float2 ml = make_float2(-INFINITY, 0.0f);
        if (lane < runs)
            ml = __ldcg(reinterpret_cast<const float2 *>(p.part_ml + (size_t)slot * p.ml_slot +
                                                         (size_t)(kvh * group + h) * p.splits * 2) + lane);
        const float big = warp_max(ml.x);
        s_ml[h][lane] = lane == kStagedRow - 1 ? make_float2(big, 0.0f)
                                               : make_float2(ml.x == -INFINITY ? 0.0f : ex2(ml.x - big), ml.y);
    }
    __syncthreads();
    for (unsigned spin = 0; !mbar_try_wait(bar, 0);)
        if (++spin > kSpinLimit) {
            landed = false;
            break;
        }
    for (int item = tid; item < group * 64; item += kThreads) {
        const int h = item >> 6;
        const float2 *const wl = s_ml[h];
        const float4 *const x = reinterpret_cast<const float4 *>(area + h * row) + (item & 63);
        Part r;
        r.a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        r.l = 0.0f;
        r.m = wl[kStagedRow - 1].x;
#pragma unroll 4
        for (int i = 0; i < runs; i++) {
            const float4 v = x[i * 64];
            const float2 w = wl[i];
            r.a.x = fmaf(v.x, w.x, r.a.x);
            r.a.y = fmaf(v.y, w.x, r.a.y);
            r.a.z = fmaf(v.z, w.x, r.a.z);
            r.a.w = fmaf(v.w, w.x, r.a.w);
            r.l = fmaf(w.y, w.x, r.l);
        }
        emit_item(p, slot, kvh, group, item, r);
    }
    return true;
}

// Which rows a CTA works on.
struct Work {
    int slot, kvh, run;   // slot < 0: none; run: index of the partial (a cluster of kC CTAs shares one)
    int runs;             // live runs of the head (what its fold reads); run >= runs: a run without rows
    int row0, row1;       // this CTA's rows; row0 a multiple of 16
    int unit;             // rows per unit of a warp: 16 while that gives every warp at most one, else 32
    int len;              // live rows of the slot
};

__device__ __forceinline__ int div_up(int a, int b) { return (a + b - 1) / b; }

// The balanced plan of one stream: every warp of every run gets a unit before any gets two, and units
// are 16 rows as long as one each is enough (half the latency of a short step), then 32 (an eighth
// fewer instructions per row). Units are counted in eights, so that neighbouring columns of a stream
// mostly share a plan; the last few can be empty.
struct Balance {
    int unit, units, runs;
};
__device__ __forceinline__ Balance balance(const DecodeParams &p, int len, int ctas, int most) {
    const int cap = min(p.splits, p.run_cap), warps = kWarps * ctas;
    Balance b;
    b.unit = div_up(len, 16) <= cap * warps ? 16 : most;
    b.units = div_up(len, 16 * 8) * 8;
    if (b.unit == 32) b.units = div_up(len, 32 * 8) * 8;
    b.runs = max(1, min(div_up(b.units, warps), cap));
    return b;
}

// Run `run` of a head under plan b; the first units % runs runs get one unit more than the others.
template <int kC>
__device__ __forceinline__ Work plan_run(const Balance &b, int slot, int kvh, int run, int rank, int len) {
    Work w;
    w.slot = slot;
    w.len = len;
    w.kvh = kvh;
    w.run = run;
    w.runs = b.runs;
    w.unit = b.unit;
    w.row0 = w.row1 = 0;
    if (run < b.runs) {
        const int each = b.units / b.runs, more = b.units - each * b.runs;
        const int c0 = run * each + min(run, more), c1 = c0 + each + (run < more ? 1 : 0);
        w.row0 = (c0 + (c1 - c0) * rank / kC) * b.unit;   // (past the end for a CTA without rows)
        w.row1 = min((c0 + (c1 - c0) * (rank + 1) / kC) * b.unit, len);
    }
    return w;
}

// One stream of `len` live rows.
template <int kC, int kUnitRows>
__device__ __forceinline__ Work plan_stream(const DecodeParams &p, int slot, int rank, int len) {
    const int cluster = (int)blockIdx.x / kC;
    if (!p.by_stride && p.run_cap > 0) {
        const int cap = min(p.splits, p.run_cap), kvh = cluster / cap;
        return plan_run<kC>(balance(p, len, kC, kUnitRows), slot, kvh, cluster - kvh * cap, rank, len);
    }
    // fixed runs of ceil(span / splits) rows, rounded up to 64
    Work w;
    w.slot = slot;
    w.len = len;
    w.kvh = cluster / p.splits;
    w.run = cluster - w.kvh * p.splits;
    w.runs = p.splits;
    const int span = p.by_stride ? p.stride : len;
    const int per = div_up(div_up(span, p.splits), kTile) * kTile;
    w.row0 = min(w.run * per, len);
    w.row1 = min(w.row0 + per, len);
    w.unit = w.row1 - w.row0 <= 16 * kWarps ? 16 : kUnitRows;
    return w;
}

}  // namespace warp_body
}  // namespace hipml
