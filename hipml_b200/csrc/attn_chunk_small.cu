// Causal chunk attention for few (query, key) pairs, head_dim 256: one launch straight from the cache.
//
// CPU definition: crates/hipml-core/src/attention.rs:56-102 per query row with seq = pos0 + t + 1.
//
// The tensor-core path (attn_chunk_tc.cu) is two launches with ~10 us of fixed cost per CTA pair, however
// short the chunk; a follow-up of a few dozen tokens to a short conversation is all latency there (37
// tokens at position 29: 19 us of staging and attention, here 8). Here a CTA of eight warps takes one
// query token and KV head; a warp takes four keys at a time for all heads of the group, reads and
// dequantises each row once, and sums the 24 dot products over the lanes by one reduce-scatter. Plain f32
// products and sums. Bound by latency, 5.4 us per 100 keys, up to about a wave of CTAs, by the CUDA cores'
// FMA rate beyond; where either passes the tensor cores' time the dispatch goes back to them (small_chunk).
// 37 tokens at 29 with their append: 26.2 -> 12.4 us.
#include "decode_rows_f32.cuh"
#include "decode_warp_body.cuh"

namespace hipml {

namespace {

using namespace warp_body;

struct SmallParams {
    const float *q;        // [tokens][n_heads * 256]
    const void *k, *v;
    float *out;
    int n_heads, n_kv, pos0, tokens, stride;
    float scale_log2;
};

// Values 8 * lane .. + 7 of one cache row.
template <int kType>   // 0 f32 position-major, 1 q8_0, 2 q4_0 head-major
__device__ __forceinline__ void load_row8(const void *cache, int n_kv, int kvh, int stride, int key, int lane,
                                          float (&x)[8]) {
    if constexpr (kType == 0) {
        const float4 *r = reinterpret_cast<const float4 *>((const float *)cache + ((size_t)key * n_kv + kvh) * 256) + 2 * lane;
        const float4 a = r[0], b = r[1];
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
        const int blk = lane >> 2, sub = lane & 3;
        const unsigned char *b = (const unsigned char *)cache +
                                 ((size_t)kvh * stride + key) * (kType == 2 ? kQ4RowBytes : kRowBytes) +
                                 blk * (kType == 2 ? kQ4BlockBytes : kQ8BlockBytes);
        const float d = half_bits_to_float(*(const unsigned short *)b);
        if constexpr (kType == 1) {
            const unsigned short *c = (const unsigned short *)(b + 2 + sub * 8);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned short w = c[j];
                x[2 * j] = d * (float)(signed char)(w & 0xff);
                x[2 * j + 1] = d * (float)(signed char)(w >> 8);
            }
        } else {
            // dims 8 * sub .. + 7 of the block: the low (sub < 2) or high nibbles of bytes 8 * (sub & 1) .. + 7
            const unsigned short *c = (const unsigned short *)(b + 2 + (sub & 1) * 8);
            const int shift = (sub >> 1) * 4;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned short w = c[j];
                x[2 * j] = d * ((float)((w >> shift) & 0xf) - 8.0f);
                x[2 * j + 1] = d * ((float)((w >> (8 + shift)) & 0xf) - 8.0f);
            }
        }
    }
}

// grid (n_kv, tokens); the last tokens, which see the most keys, start first.
template <int kType, int kHeads>
__global__ void __launch_bounds__(kThreads, 2) attn_chunk_small(SmallParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) float s_q[8 * 256];
    __shared__ __align__(16) float s_w[kWarps][8][kRowsAtOnce];
    __shared__ float2 s_ml[8 * kWarps];
    griddep_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = blockIdx.x, token = p.tokens - 1 - (int)blockIdx.y, group = p.n_heads / p.n_kv;
    const int seq = p.pos0 + token + 1;
    griddep_wait();
    for (int i = tid; i < 8 * 64; i += kThreads) {
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < group * 64) x = reinterpret_cast<const float4 *>(p.q + ((size_t)token * p.n_heads + kvh * group) * 256)[i];
        x.x *= p.scale_log2;
        x.y *= p.scale_log2;
        x.z *= p.scale_log2;
        x.w *= p.scale_log2;
        reinterpret_cast<float4 *>(s_q)[i] = x;
    }
    __syncthreads();
    RowsF32<kHeads> st;
    st.start();
    for (int r0 = warp * kRowsAtOnce; r0 < seq; r0 += kWarps * kRowsAtOnce) {
        float k[kRowsAtOnce][8], v[kRowsAtOnce][8];
#pragma unroll
        for (int r = 0; r < kRowsAtOnce; r++) {
            const int key = min(r0 + r, seq - 1);
            load_row8<kType>(p.k, p.n_kv, kvh, p.stride, key, lane, k[r]);
            load_row8<kType>(p.v, p.n_kv, kvh, p.stride, key, lane, v[r]);
        }
        st.add(k, v, s_q + 8 * lane, s_q + 8 * lane + 4, s_w[warp], r0, seq, lane);
    }
    st.finish(s_ml, warp, lane);
    float *const mine = reinterpret_cast<float *>(smem) + warp * 8 * kHeadPitch + 8 * lane;
#pragma unroll
    for (int h = 0; h < kHeads; h++) {
        *reinterpret_cast<float4 *>(mine + h * kHeadPitch) = make_float4(st.acc[h][0], st.acc[h][1], st.acc[h][2], st.acc[h][3]);
        *reinterpret_cast<float4 *>(mine + h * kHeadPitch + 4) =
            make_float4(st.acc[h][4], st.acc[h][5], st.acc[h][6], st.acc[h][7]);
    }
    __syncthreads();
    fold_warps(smem, 8 * kHeadPitch * 4, s_ml, group * 64, [&](int item, const Part &r) {
        float4 y;
        y.x = __fdiv_rn(r.a.x, r.l);
        y.y = __fdiv_rn(r.a.y, r.l);
        y.z = __fdiv_rn(r.a.z, r.l);
        y.w = __fdiv_rn(r.a.w, r.l);
        reinterpret_cast<float4 *>(p.out + ((size_t)token * p.n_heads + kvh * group) * 256)[item] = y;
    });
}

template <int kType, int kHeads>
int launch(cudaStream_t stream, const SmallParams &p) {
    constexpr int kSmem = kWarps * 8 * kHeadPitch * 4;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const cudaError_t e =
            cudaFuncSetAttribute(attn_chunk_small<kType, kHeads>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    return launch_pdl(attn_chunk_small<kType, kHeads>, dim3(p.n_kv, p.tokens), dim3(kThreads), (size_t)kSmem, stream, 1, p);
}

}  // namespace

int launch_chunk_small(cudaStream_t stream, const float *q, const void *k_cache, const void *v_cache, float *out,
                       int n_heads, int n_kv, int kv_dtype, int stride, int pos0, int tokens) {
    const SmallParams p = {q, k_cache, v_cache, out, n_heads, n_kv, pos0, tokens, stride,
                           (1.0f / sqrtf(256.0f)) * 1.4426950408889634f};
    const bool six = n_heads / n_kv <= 6;
    if (kv_dtype == 0) return six ? launch<0, 6>(stream, p) : launch<0, 8>(stream, p);
    if (kv_dtype == 1) return six ? launch<1, 6>(stream, p) : launch<1, 8>(stream, p);
    return six ? launch<2, 6>(stream, p) : launch<2, 8>(stream, p);
}

}  // namespace hipml
