// Split-K decode over the f32 position-major cache for 1..R consecutive columns, and the
// matching multi-row append.
//
// CPU definition: crates/hipml-core/src/attention.rs:56-102 with seq = pos0 + c + 1 for
// column c. Kernels replaced: crates/hipml-kernels/kernels/attn_decode_cols_f32.hip:31-213
// (split pass + reduce) and kv_append_cols_f32.hip:11-31; launcher
// crates/hipml-kernels/src/attn_gpu/imp/attn_cols.rs:15-173. The key axis is cut into
// `splits` runs of `per = ceil(n_ctx / splits)` rows fixed in cache positions, so a column's
// arithmetic does not depend on how many columns share the launch. This is the `--kv f32` path of the
// reference: plain f32 products and sums on the CUDA cores.
//
// head_dim 256: attn_decode_rows_f32, a CTA per (run, KV head, column). Bound by the HBM stream of the
// rows (16.8 MB per layer at 2,048 rows) once latency is hidden; the arithmetic is 1.5 FMA per byte. So a
// warp reads a row once for all heads of the group (one warp per head read it six times), four rows at
// a time with all loads in flight; the four rows' dot products are summed over the lanes by one
// reduce-scatter (25 shuffles for 24 sums, where a butterfly each took 120). Other head sizes:
// attn_decode_cols_f32, one warp per (query head, run, column).
#include <atomic>

#include "decode_rows_f32.cuh"

namespace hipml {

struct ColsParams {
    const float *q;        // [rows][n_heads*head_dim]
    const float *k;        // [n_ctx][n_kv*head_dim]
    const float *v;
    float *part_acc;       // [rows][n_heads][splits][head_dim]
    float *part_ml;        // [rows][n_heads][splits][2]
    int n_heads, n_kv, head_dim;
    int pos0, rows;
    float scale_log2;
    int splits, per;
};

namespace {

using namespace warp_body;

constexpr int kOffMlF32 = kWarps * 8 * kHeadPitch * 4;             // after the warps' partials: [8 heads][warp]
constexpr int kOffInF32 = kOffMlF32 + kWarps * 8 * 8;              // partials of the cluster's CTAs
constexpr int kOffInMlF32 = kOffInF32 + 8 * 256 * 4;
constexpr int kOffBarF32 = kOffInMlF32 + 8 * 8 * 8;
constexpr int kSmemF32 = kOffBarF32 + 8;

__device__ int g_arrive_f32[kArriveRegions * kArriveRegionInts];

// kC: CTAs (runs) per cluster, each sent its slice of the others' partials to fold. grid (n_kv * clusters * kC,
// columns). d: out, scratch and counters (as the quantised body's).
template <int kHeads, int kC>
__global__ void __launch_bounds__(kThreads, 2) attn_decode_rows_f32(ColsParams p, DecodeParams d, int clusters, int *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) float s_q[8 * 256];
    __shared__ __align__(16) float s_w[kWarps][8][kRowsAtOnce];
    __shared__ int s_last;
    griddep_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank(), cluster = (int)blockIdx.x / kC;
    const int kvh = cluster / clusters, in_head = cluster - kvh * clusters, col = blockIdx.y;
    const int group = p.n_heads / p.n_kv, width = p.n_kv * 256, seq = p.pos0 + col + 1;
    const int items = group * 64;
    const unsigned bar_in = smem_u32(smem + kOffBarF32);
    if (tid == 0) {
        mbar_init(bar_in, 1);
        mbar_init_fence();
        mbar_arrive_expect_tx(bar_in, inbox_bytes<kC>(items, rank));
    }
    cluster_arrive();   // (waited for before anything is sent to another CTA)
    // this warp's share of the run, fixed in cache positions, cut at the column's last row
    const int run = in_head * kC + rank;
    const int run0 = run * p.per, run_rows = run < p.splits ? p.per : 0;
    const int lo = min(run0 + run_rows * warp / kWarps, seq), hi = min(run0 + run_rows * (warp + 1) / kWarps, seq);
    const float *const kb = p.k + (size_t)kvh * 256, *const vb = p.v + (size_t)kvh * 256;
    // (asks L2 only; the rows are read once the grids ahead are done)
    for (int i = lane; i < 2 * (hi - lo); i += 32)
        prefetch_l2(((i & 1) ? vb : kb) + (size_t)(lo + (i >> 1)) * width, 1024);
    if (tid == 0) ask_l2(p.q + ((size_t)col * p.n_heads + kvh * group) * 256, 1024LL * group);
    griddep_wait();
    cluster_wait();
    for (int i = tid; i < 8 * 64; i += kThreads) {
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < group * 64)
            x = reinterpret_cast<const float4 *>(p.q + ((size_t)col * p.n_heads + kvh * group) * 256)[i];
        x.x *= p.scale_log2;
        x.y *= p.scale_log2;
        x.z *= p.scale_log2;
        x.w *= p.scale_log2;
        reinterpret_cast<float4 *>(s_q)[i] = x;
    }
    __syncthreads();

    // lane: dims 4 * lane .. + 3 and 128 + 4 * lane .. + 3
    RowsF32<kHeads> st;
    st.start();
    for (int r0 = lo; r0 < hi; r0 += kRowsAtOnce) {
        float k[kRowsAtOnce][8], v[kRowsAtOnce][8];
#pragma unroll
        for (int r = 0; r < kRowsAtOnce; r++) {
            const size_t at = (size_t)min(r0 + r, hi - 1) * width + 4 * lane;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float4 a = *reinterpret_cast<const float4 *>(kb + at + 128 * i);
                const float4 b = *reinterpret_cast<const float4 *>(vb + at + 128 * i);
                k[r][4 * i] = a.x; k[r][4 * i + 1] = a.y; k[r][4 * i + 2] = a.z; k[r][4 * i + 3] = a.w;
                v[r][4 * i] = b.x; v[r][4 * i + 1] = b.y; v[r][4 * i + 2] = b.z; v[r][4 * i + 3] = b.w;
            }
        }
        st.add(k, v, s_q + 4 * lane, s_q + 128 + 4 * lane, s_w[warp], r0, hi, lane);
    }

    // ---- merge: the warps, the cluster, then the head's clusters (the last to arrive)
    float2 *const wml = reinterpret_cast<float2 *>(smem + kOffMlF32);
    st.finish(wml, warp, lane);
    float *const mine = reinterpret_cast<float *>(smem) + warp * 8 * kHeadPitch;
#pragma unroll
    for (int h = 0; h < kHeads; h++) {
        *reinterpret_cast<float4 *>(mine + h * kHeadPitch + 4 * lane) = make_float4(st.acc[h][0], st.acc[h][1], st.acc[h][2], st.acc[h][3]);
        *reinterpret_cast<float4 *>(mine + h * kHeadPitch + 128 + 4 * lane) =
            make_float4(st.acc[h][4], st.acc[h][5], st.acc[h][6], st.acc[h][7]);
    }
    __syncthreads();
    float4 *const inbox = reinterpret_cast<float4 *>(smem + kOffInF32);
    float2 *const inbox_ml = reinterpret_cast<float2 *>(smem + kOffInMlF32);
    fold_warps(smem, 8 * kHeadPitch * 4, wml, items, [&](int item, const Part &r) {
        send_item<kC>(inbox, inbox_ml, bar_in, items, rank, item, r);
    });
    if (!await_inbox(bar_in, 0) && status) atomicCAS(status, 0, 21);
    const bool one = clusters == 1 && d.out != nullptr;
    fold_inbox<kC>(inbox, inbox_ml, items, rank, [&](int item, const Part &r) {
        if (one) {
            emit_item(d, col, kvh, group, item, r);
            return;
        }
        const size_t row = (size_t)(kvh * group + (item >> 6)) * d.splits + in_head;
        reinterpret_cast<float4 *>(d.part_acc + (size_t)col * d.acc_slot + row * 256)[item & 63] = r.a;
        if (writes_pair<kC>(items, rank, item))
            *reinterpret_cast<float2 *>(d.part_ml + (size_t)col * d.ml_slot + row * 2) = make_float2(r.m, r.l);
    });
    if (d.out != nullptr && !one) {
        int *const ctr = g_arrive_f32 + (size_t)d.arrive_region * kArriveRegionInts +
                         (size_t)(col * p.n_kv + kvh) * kC + rank;
        __syncthreads();
        if (tid == 0) {
            const int last = arrive_acq_rel(ctr) == clusters - 1;
            if (last) *ctr = 0;
            s_last = last;
        }
        __syncthreads();
        if (s_last) fold_runs<kC, 8>(d, col, kvh, group, clusters, rank, nullptr);
    }
}

// One warp per (query head, run, column), any head size.
__global__ void __launch_bounds__(128) attn_decode_cols_f32(ColsParams p) {
    griddep_launch();
    griddep_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int col = blockIdx.y;
    if (warp >= p.n_heads * p.splits) return;
    const int h = warp / p.splits, split = warp - h * p.splits;
    const int kvh = h / (p.n_heads / p.n_kv);
    const int live = lane * 8 < p.head_dim;
    const int d0 = lane * 8;
    const int width = p.n_kv * p.head_dim;
    const int seq = p.pos0 + col + 1;
    const int lo = min(split * p.per, seq), hi = min(lo + p.per, seq);

    float qv[8];
    const float *q = p.q + ((size_t)col * p.n_heads + h) * p.head_dim;
#pragma unroll
    for (int j = 0; j < 8; j++) qv[j] = live ? q[d0 + j] * p.scale_log2 : 0.0f;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float m = -INFINITY, l = 0.0f;
    for (int pos = lo; pos < hi; pos++) {
        const size_t at = (size_t)pos * width + kvh * p.head_dim + d0;
        float part = 0.0f;
        if (live) {
#pragma unroll
            for (int j = 0; j < 8; j++) part += qv[j] * p.k[at + j];
        }
        const float s = warp_sum(part);
        const float m_new = fmaxf(m, s);
        const float corr = exp2f(m - m_new);
        const float w = exp2f(s - m_new);
        l = l * corr + w;
        m = m_new;
        if (live) {
#pragma unroll
            for (int j = 0; j < 8; j++) acc[j] = acc[j] * corr + w * p.v[at + j];
        }
    }
    const size_t slot = ((size_t)col * p.n_heads + h) * p.splits + split;
    if (live) {
#pragma unroll
        for (int j = 0; j < 8; j++) p.part_acc[slot * p.head_dim + d0 + j] = acc[j];
    }
    if (lane == 0) {
        p.part_ml[slot * 2] = m;
        p.part_ml[slot * 2 + 1] = l;
    }
}

}  // namespace

// Entry name, parameter list and linear launch shape of the reference's kernel: row c of k/v
// lands at cache row pos0 + c; threads [0,width) of a row copy K, [width,2*width) copy V.
extern "C" __global__ void kv_append_cols_f32(float *__restrict__ k_cache,
                                              float *__restrict__ v_cache,
                                              const float *__restrict__ k,
                                              const float *__restrict__ v, int pos0, int rows,
                                              int width) {
    griddep_launch();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2LL * width * rows) return;
    const int c = (int)(i / (2 * width));
    const int j = (int)(i - (long long)c * 2 * width);
    if ((threadIdx.x & 31) == 0)   // a warp's 32 floats, as far as they are of the same row
        ask_l2(j < width ? k + (size_t)c * width + j : v + (size_t)c * width + j - width,
               4LL * min(32, j < width ? width - j : 2 * width - j));
    griddep_wait();
    const size_t base = (size_t)(pos0 + c) * width;
    if (j < width)
        k_cache[base + j] = k[(size_t)c * width + j];
    else
        v_cache[base + j - width] = v[(size_t)c * width + j - width];
}

const void *lookup_cols_kernel(const char *name) {
    if (strcmp(name, "kv_append_cols_f32") == 0) return (const void *)kv_append_cols_f32;
    return nullptr;
}

namespace {

template <int kHeads, int kC>
int launch_rows_f32_heads(cudaStream_t stream, const ColsParams &p, const DecodeParams &d, int clusters) {
    static std::atomic<int *> status_word[64] = {};   // nullptr: device not set up yet
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    int *status = status_word[dev].load(std::memory_order_acquire);
    if (status == nullptr) {
        const cudaError_t e =
            cudaFuncSetAttribute(attn_decode_rows_f32<kHeads, kC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemF32);
        if (e != cudaSuccess) return (int)e;
        status = device_status_word();
        if (status == nullptr) return launch_status();
        status_word[dev].store(status, std::memory_order_release);
    }
    return launch_pdl(attn_decode_rows_f32<kHeads, kC>, dim3(p.n_kv * clusters * kC, p.rows), dim3(kThreads),
                      (size_t)kSmemF32, stream, kC, p, d, clusters, status);
}

int launch_rows_f32(cudaStream_t stream, const ColsParams &p, float *out, long long acc_slot, long long ml_slot,
                    long long out_slot) {
    // one cluster of eight where that is all the runs (114 rows: 6.8 us a layer, with append, against 8.2 in two of
    // four), else clusters of four, which fill the device better (2,048 rows: 15.7 -> 12.7 us)
    const int size = p.splits <= 8 ? 8 : 4, clusters = (p.splits + size - 1) / size;
    DecodeParams d = {};
    d.part_acc = p.part_acc;
    d.part_ml = p.part_ml;
    d.n_heads = p.n_heads;
    d.n_kv = p.n_kv;
    d.head_dim = 256;
    d.splits = p.splits;
    d.acc_slot = acc_slot;
    d.ml_slot = ml_slot;
    d.out = out;
    d.out_slot = out_slot;
    d.out_head_stride = 256;
    d.normalize = 1;
    d.arrive_region = decode_arrive_region(stream, (long long)p.rows * p.n_kv * size);
    const bool second_launch = d.arrive_region < 0;
    if (second_launch) d.out = nullptr;
    const bool six = p.n_heads / p.n_kv <= 6;
    const int rc = size == 8 ? (six ? launch_rows_f32_heads<6, 8>(stream, p, d, clusters)
                                    : launch_rows_f32_heads<8, 8>(stream, p, d, clusters))
                             : (six ? launch_rows_f32_heads<6, 4>(stream, p, d, clusters)
                                    : launch_rows_f32_heads<8, 4>(stream, p, d, clusters));
    if (rc != 0 || !second_launch) return rc;
    FoldParams f = {};
    f.acc = p.part_acc;
    f.ml = p.part_ml;
    f.out = out;
    f.head_dim = 256;
    f.splits = clusters;
    f.acc_head_stride = (long long)p.splits * 256;
    f.acc_split_stride = 256;
    f.ml_head_stride = (long long)p.splits * 2;
    f.ml_split_stride = 2;
    f.acc_slot = acc_slot;
    f.ml_slot = ml_slot;
    f.out_slot = out_slot;
    f.out_head_stride = 256;
    f.normalize = 1;
    return launch_decode_fold(stream, f, p.n_heads, p.rows);
}

}  // namespace

int launch_decode_cols_f32(cudaStream_t stream, const float *q, const float *k, const float *v,
                           float *part_acc, float *part_ml, float *out, int n_heads, int n_kv,
                           int head_dim, int n_ctx, int pos0, int rows, int splits) {
    ColsParams p;
    p.q = q;
    p.k = k;
    p.v = v;
    p.part_acc = part_acc;
    p.part_ml = part_ml;
    p.n_heads = n_heads;
    p.n_kv = n_kv;
    p.head_dim = head_dim;
    p.pos0 = pos0;
    p.rows = rows;
    p.scale_log2 = (1.0f / sqrtf((float)head_dim)) * 1.4426950408889634f;
    p.splits = splits;
    p.per = (n_ctx + splits - 1) / splits;
    const long long acc_slot = (long long)n_heads * splits * head_dim, ml_slot = (long long)n_heads * splits * 2;
    const long long out_slot = (long long)n_heads * head_dim;
    const size_t align = reinterpret_cast<size_t>(q) | reinterpret_cast<size_t>(k) | reinterpret_cast<size_t>(v) |
                         reinterpret_cast<size_t>(part_acc) | reinterpret_cast<size_t>(out);
    if (head_dim == 256 && (align & 15) == 0 && (reinterpret_cast<size_t>(part_ml) & 7) == 0)
        return launch_rows_f32(stream, p, out, acc_slot, ml_slot, out_slot);
    dim3 grid((n_heads * splits + 3) / 4, rows);
    if (int e = launch_pdl(attn_decode_cols_f32, grid, dim3(128), 0, stream, 1, p)) return e;
    if (int e = launch_status()) return e;
    return launch_decode_reduce(stream, part_acc, part_ml, out, n_heads, head_dim, splits, rows, acc_slot, ml_slot,
                                out_slot);
}

}  // namespace hipml
