// Attention of one query group over f32 values of cache rows on the CUDA cores, a warp at a time: shared
// by the f32-cache decode (attn_decode_f32.cu) and the small chunks (attn_chunk_small.cu). head_dim 256; a
// lane owns eight dims of every row, four rows are taken together.
#pragma once

#include "decode_warp_body.cuh"

namespace hipml {
namespace warp_body {

constexpr int kRowsAtOnce = 4;

// Sums v[row][head] over the 32 lanes; lane 8 * row + head returns its own sum (25 shuffles for 24 sums).
template <int kHeads>
__device__ __forceinline__ float reduce_scatter(const float (&v)[kRowsAtOnce][kHeads], int lane) {
    float a[2][kHeads], b[8];
#pragma unroll
    for (int h = 0; h < kHeads; h++) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float keep = (lane & 16) ? v[2 + r][h] : v[r][h], give = (lane & 16) ? v[r][h] : v[2 + r][h];
            a[r][h] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
        }
        const float keep = (lane & 8) ? a[1][h] : a[0][h], give = (lane & 8) ? a[0][h] : a[1][h];
        b[h] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
#pragma unroll
    for (int h = kHeads; h < 8; h++) b[h] = 0.0f;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int h = 0; h < o; h++) {
            const float keep = (lane & o) ? b[o + h] : b[h], give = (lane & o) ? b[h] : b[o + h];
            b[h] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    return b[0];
}

template <int kHeads>
struct RowsF32 {
    float acc[kHeads][8];
    float m, l;   // lane 8 * row + head: the head's maximum, the sum over rows = row (mod 4)

    __device__ __forceinline__ void start() {
#pragma unroll
        for (int h = 0; h < kHeads; h++)
#pragma unroll
            for (int e = 0; e < 8; e++) acc[h][e] = 0.0f;
        m = -INFINITY;
        l = 0.0f;
    }
    // Rows r0 .. r0 + 3 (those from `end` on weigh nothing; at least one lies before it). q0, q1: the lane's dims
    // 0..3 and 4..7 of head 0's scaled query, heads 256 floats apart; w_at: the warp's [8][4] exchange.
    __device__ __forceinline__ void add(const float (&k)[kRowsAtOnce][8], const float (&v)[kRowsAtOnce][8], const float *q0,
                                        const float *q1, float (*w_at)[kRowsAtOnce], int r0, int end, int lane) {
        float s[kRowsAtOnce][kHeads];
#pragma unroll
        for (int h = 0; h < kHeads; h++) {
            const float4 a = *reinterpret_cast<const float4 *>(q0 + h * 256);
            const float4 b = *reinterpret_cast<const float4 *>(q1 + h * 256);
#pragma unroll
            for (int r = 0; r < kRowsAtOnce; r++) {
                float x = a.x * k[r][0];
                x = fmaf(a.y, k[r][1], x);
                x = fmaf(a.z, k[r][2], x);
                x = fmaf(a.w, k[r][3], x);
                x = fmaf(b.x, k[r][4], x);
                x = fmaf(b.y, k[r][5], x);
                x = fmaf(b.z, k[r][6], x);
                s[r][h] = fmaf(b.w, k[r][7], x);
            }
        }
        float score = reduce_scatter<kHeads>(s, lane);
        if (r0 + (lane >> 3) >= end) score = -INFINITY;
        float top = fmaxf(score, __shfl_xor_sync(0xffffffffu, score, 8));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
        const float m_new = fmaxf(m, top);
        if (__any_sync(0xffffffffu, m_new > m)) {
            const float corr = ex2(m - m_new);
            l *= corr;
            m = m_new;
#pragma unroll
            for (int h = 0; h < kHeads; h++) {
                const float c = __shfl_sync(0xffffffffu, corr, h);
#pragma unroll
                for (int e = 0; e < 8; e++) acc[h][e] *= c;
            }
        }
        const float w = ex2(score - m);
        l += w;
        w_at[lane & 7][lane >> 3] = w;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < kHeads; h++) {
            const float4 wh = *reinterpret_cast<const float4 *>(w_at[h]);
            const float wr[4] = {wh.x, wh.y, wh.z, wh.w};
#pragma unroll
            for (int r = 0; r < kRowsAtOnce; r++)
#pragma unroll
                for (int e = 0; e < 8; e++) acc[h][e] = fmaf(wr[r], v[r][e], acc[h][e]);
        }
        __syncwarp();
    }
    // The warp's {maximum, sum} of every head into ml[head][warp].
    __device__ __forceinline__ void finish(float2 *ml, int warp, int lane) {
        l += __shfl_xor_sync(0xffffffffu, l, 8);
        l += __shfl_xor_sync(0xffffffffu, l, 16);
        if (lane < 8) ml[lane * kWarps + warp] = make_float2(m, l);
    }
};

}  // namespace warp_body
}  // namespace hipml
