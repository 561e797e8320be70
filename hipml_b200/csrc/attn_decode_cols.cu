// Split-K flash-decode of several columns of one q8_0 stream (a speculative draft's columns, head_dim 256):
// the body of attn_decode_warps.cu with the columns side by side. CPU definition per column:
// crates/hipml-core/src/ops.rs:449-518; launcher replaced: launch_kv::launch_cols_ptrs.
//
// The columns see the same rows but for the last few, so a warp loads and converts a unit's codes once
// and runs every column's MMAs on them: of the ~635 warp instructions that 16 rows cost a column, ~430
// are the codes' and only ~205 the column's own. What does not fit is the accumulators (64 a lane and
// column): they live in tensor memory, 128 of its columns per decode column, and come to the registers
// 16 at a time for the pair of blocks at hand (tcgen05.ld / st, 2 x 64 words a lane per unit).
// One launch per layer takes up to four columns in the time of about two; 4 columns of 8,192 rows took
// 36 us a layer as four grids of the single-column body.
//
// Each column's arithmetic is that of its own launch, operation for operation -- the plan, the order of
// every sum, the movements of the references -- so its result is the same bits.
#include <mutex>

#include "decode_warp_body.cuh"

namespace hipml {

namespace {

using namespace warp_body;

constexpr int kCols = 4;          // columns side by side
constexpr int kUnitRows = 32;
constexpr unsigned kTmemCols = 512;
constexpr int kMaxCols = 32;      // of a launch

struct Cfg {
    static constexpr int kSlot = kUnitRows * kRowBytes;
    static constexpr int kRing = 2 * kSlot;                        // per warp: a unit of K and one of V; later two partials
    static constexpr int kPartial = 8 * kHeadPitch * 4;
    static_assert(kRing >= 2 * kPartial, "a warp's partials fit its ring");
    static constexpr int kQBytes = 16 * 32 * 16;                   // a column's query fragments, later its partial of the CTA
    static constexpr int kBiasBytes = 8 * 4 * 16;
    static constexpr int kOffQ = kWarps * kRing;
    static constexpr int kOffBias = kOffQ + kCols * kQBytes;
    static constexpr int kOffMl = kOffBias + kCols * kBiasBytes;   // two columns' [8 heads][warps] {reference, sum}
    static constexpr int kOffCml = kOffMl + 2 * kWarps * 8 * 8;    // per column [8 heads]
    static constexpr int kOffBar = kOffCml + kCols * 8 * 8;
    static constexpr int kOffFold = kOffBar + kWarps * 2 * 8 + 8;  // weights of the last fold, after its barrier
    static constexpr int kSmem = kOffFold + kCols * 5 * kStagedRow * 8;
    static_assert(kSmem + 1024 <= 227 * 1024, "one CTA per SM");
};

__device__ int g_arrive_cols[kArriveRegions * kArriveRegionInts];

// Which columns a cluster takes. Neighbouring columns with the same plan (the same units for every warp), at
// most `each` of them, are a group; a cluster has run `run` of groups `group`, `group` + `hop`, ... Groups go
// to clusters of their own while a head has clusters to spare for their runs, and columns share conversions
// beyond (4 columns of 300 rows take 2 runs each: 8 clusters of the head's 18; of 8,192 rows 17: one cluster
// per run takes all four). `cap`: the clusters of a head; what its groups do not need ends at once, so there is one
// round of them and they take the groups in turn.
struct Share {
    int each, run, group, hop;
    unsigned starts;   // bit c: column c's plan is not column c - 1's
};
template <int kC>
__device__ __forceinline__ Share share_columns(const DecodeParams &p, int cap, int in_head, const int *len) {
    const int c = threadIdx.x & 31;
    const bool on = c < p.n_slots;
    Balance b = {0, 0, 1};
    if (on) b = balance(p, len[c], kC, kUnitRows);
    const int units = __shfl_up_sync(0xffffffffu, b.units, 1), unit = __shfl_up_sync(0xffffffffu, b.unit, 1);
    const int before = __shfl_up_sync(0xffffffffu, b.runs, 1);
    const int runs = __reduce_max_sync(0xffffffffu, b.runs);
    const int side = cap / runs;   // groups side by side, >= 1
    Share s;
    s.starts = __ballot_sync(0xffffffffu, on && (c == 0 || units != b.units || unit != b.unit || before != b.runs));
    s.each = min(kCols, div_up(p.n_slots, side));
    s.run = in_head % runs;
    s.group = in_head < side * runs ? in_head / runs : p.n_slots;
    s.hop = side;
    return s;
}
// Columns [base, end) of group s.group (none past the last); returns how many groups there are.
__device__ __forceinline__ int find_group(const Share &s, int cols, int &base, int &end) {
    base = end = cols;
    int groups = 0;
    for (int first = 0; first < cols; groups++) {
        const unsigned later = first < 31 ? s.starts >> (first + 1) : 0;
        const int last = min(min(first + s.each, cols), later ? first + __ffs(later) : cols);
        if (groups == s.group) {
            base = first;
            end = last;
        }
        first = last;
    }
    return groups;
}

// grid (n_kv * run_cap * kC), clusters of kC as in the single-column form.
template <int kC>
__global__ void __launch_bounds__(kThreads, 1) attn_decode_cols(DecodeParams p, int *status) {
    using C = Cfg;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_last;
    __shared__ unsigned s_tmem;
    __shared__ int s_len[kMaxCols];
    griddep_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int group = p.n_heads / p.n_kv;
    const int rank = (int)cluster_rank();
    unsigned char *const ring = smem + warp * C::kRing;
    const unsigned ring_addr = smem_u32(ring), bar = smem_u32(smem + C::kOffBar) + warp * 16;
    const unsigned bar_fold = smem_u32(smem + C::kOffFold) - 8;
    if (lane == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 1);
        if (warp == 0) mbar_init(bar_fold, 1);
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc<1>(smem_u32(&s_tmem), kTmemCols);
    const int cap = p.run_cap, cluster = (int)blockIdx.x / kC;
    const int kvh = cluster / cap, in_head = cluster - kvh * cap;
    // Nothing that the grids ahead may write can be relied on before they are done, but the lengths as they
    // stand are a good guess: enough to plan with and to ask L2 for the first rows. They are checked below.
    auto read_len = [&]() {   // of column tid < n_slots
        return live_len(p, __ldcg(p.len + p.len_offset + tid * p.len_stride));
    };
    if (tid < p.n_slots) s_len[tid] = read_len();
    __syncthreads();
    const size_t head_byte = (size_t)kvh * p.stride * kRowBytes;   // (the columns share the cache)
    Share sh = share_columns<kC>(p, cap, in_head, s_len);
    int base, end;
    int groups = find_group(sh, p.n_slots, base, end);
    int n, len[kCols], first, row1, nw;
    bool live;
    Work w;
    size_t step;
    const unsigned char *kp, *vp;
    auto plan = [&]() {
        live = false;
        nw = 0;
        n = end - base;
        if (n == 0) return;
        const Balance b0 = balance(p, s_len[base], kC, kUnitRows);
        int longest = 0;
#pragma unroll
        for (int c = 0; c < kCols; c++) {
            len[c] = c < n ? s_len[base + c] : 0;
            longest = max(longest, len[c]);
        }
        w = plan_run<kC>(b0, base, kvh, sh.run, rank, longest);
        live = w.run < w.runs;
        first = w.row0 + w.unit * warp;
        row1 = w.row1;
        nw = live && first < row1 ? div_up(row1 - first, w.unit * kWarps) : 0;
        step = (size_t)w.unit * kWarps * kRowBytes;
        kp = p.k + head_byte + (size_t)first * kRowBytes;
        vp = p.v + head_byte + (size_t)first * kRowBytes;
    };
    auto unit_bytes = [&](int i) { return (unsigned)(min(w.unit, row1 - (first + i * w.unit * kWarps)) * kRowBytes); };
    auto fetch = [&](int i, const unsigned char *src, int slot) {   // unit i: one lane
        const unsigned bytes = unit_bytes(i);
        mbar_arrive_expect_tx(bar + 8 * slot, bytes);
        bulk_load(ring_addr + slot * C::kSlot, src, bytes, bar + 8 * slot);
    };
    plan();
    if (lane == 0 && nw > 0) {
        prefetch_l2(kp, unit_bytes(0));
        prefetch_l2(vp, unit_bytes(0));
    }
    griddep_wait();
    unsigned phase = 0, fold_phase = 0;
    bool landed = true, checked = false;
    auto wait = [&](int slot) {
        unsigned spin = 0;
        while (!mbar_try_wait(bar + 8 * slot, phase)) {
            if (++spin > kSpinLimit) {   // the copy never landed: flag it and carry on
                landed = false;
                break;
            }
        }
    };

    for (;;) {
        const int real_len = !checked && tid < p.n_slots ? read_len() : 0;
        // Query fragments of every column, warp b makes block b's (as in the single-column body).
        float2 x[kCols][2][2];
#pragma unroll
        for (int c = 0; c < kCols; c++) {
            const float *const qh = p.q + (size_t)(base + c) * p.q_slot + (size_t)(kvh * group + g) * 256;
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    x[c][k][i] = make_float2(0.0f, 0.0f);
                    if (g < group && c < n)
                        x[c][k][i] = *reinterpret_cast<const float2 *>(qh + k_word_dim(warp, 4 * k + t, 2 * i));
                }
        }
        if (lane == 0 && nw > 0) {
            fetch(0, kp, 0);
            fetch(0, vp, 1);
        }
#pragma unroll
        for (int c = 0; c < kCols; c++)
            if (c < n)
                store_query<false>(x[c], p.scale_log2, warp, lane, reinterpret_cast<uint4 *>(smem + C::kOffQ + c * C::kQBytes),
                                   reinterpret_cast<float *>(smem + C::kOffBias + c * C::kBiasBytes));
        tc_fence_before();
        if (checked) {
            __syncthreads();
        } else if (__syncthreads_or(tid < p.n_slots && real_len != s_len[tid])) {
            // Rare: the lengths changed after they were first looked at. What was fetched lands, unused (its
            // slots' barriers start over), and the CTA plans again.
            if (lane == 0 && nw > 0) {
                for (int i = 0; i < 2; i++) {
                    for (unsigned spin = 0; !mbar_try_wait(bar + 8 * i, 0) && spin < kSpinLimit; spin++) {}
                    mbar_inval(bar + 8 * i);
                    mbar_init(bar + 8 * i, 1);
                }
                mbar_init_fence();
            }
            if (tid < p.n_slots) s_len[tid] = real_len;
            __syncthreads();
            sh = share_columns<kC>(p, cap, in_head, s_len);
            groups = find_group(sh, p.n_slots, base, end);
            plan();
            checked = true;
            continue;
        }
        checked = true;
        tc_fence_after();
        if (base >= p.n_slots) break;
        if (live) {
        // this warp's accumulators of column c: lanes 32 * (warp % 4), columns 128 c + 64 * (warp / 4)
        const unsigned tmem = s_tmem + ((unsigned)(warp & 3) << 21) + 64u * (warp >> 2);

        Running run[kCols];
#pragma unroll
        for (int c = 0; c < kCols; c++) start(run[c]);
        auto work = [&](auto tiles, int i, int rows) __attribute__((always_inline)) {
            constexpr int kT = decltype(tiles)::value;
            const int r0 = first + i * w.unit * kWarps;
            // ---- scores of all columns
            wait(0);
            float s[kCols][kT][4];
#pragma unroll
            for (int c = 0; c < kCols; c++)
#pragma unroll
                for (int j = 0; j < kT; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++) s[c][j][e] = 0.0f;
            const unsigned *const krow = reinterpret_cast<const unsigned *>(ring) + g * Row<false>::kPitch;
            auto score = [&](auto m) __attribute__((always_inline)) {
                constexpr int M = decltype(m)::value;
                KFrag<kT> f;
                load_k<M, false, kT>(krow, t, f);
#pragma unroll
                for (int c = 0; c < kCols; c++)
                    if (c < n)
                        add_scores<M, kT>(f, reinterpret_cast<const uint4 *>(smem + C::kOffQ + c * C::kQBytes) + lane,
                                          reinterpret_cast<const float4 *>(smem + C::kOffBias + c * C::kBiasBytes) + t, s[c]);
            };
            score(Int<0>{});
            score(Int<1>{});
            score(Int<2>{});
            score(Int<3>{});
            __syncwarp();
            kp += step;
            if (lane == 0 && i + 1 < nw) fetch(i + 1, kp, 0);
            // ---- softmax
            __half2 ph[kCols][kT][2], pl[kCols][kT][2];
#pragma unroll
            for (int c = 0; c < kCols; c++) {
                if (c >= n) break;
                const int rows_c = min(w.unit, min(row1, len[c]) - r0);
                if (rows_c <= 0) {   // the unit begins past this column's end: it adds nothing
#pragma unroll
                    for (int j = 0; j < kT; j++)
#pragma unroll
                        for (int e = 0; e < 2; e++) ph[c][j][e] = pl[c][j][e] = __float2half2_rn(0.0f);
                    continue;
                }
                float corr[2];
                if (softmax<kT>(s[c], rows_c, g, run[c], ph[c], pl[c], corr) && i > 0) {
#pragma unroll 1
                    for (int m = 0; m < 4; m++) {
                        float a[16];
                        tmem_ld16(tmem + 128 * c + 16 * m, a);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; e++) a[e] *= corr[e & 1];
                        tmem_st16(tmem + 128 * c + 16 * m, a);
                    }
                    tmem_wait_st();
                }
            }
            // ---- values
            wait(1);
            unsigned char *const vt = ring + C::kSlot;
            // rows past the end have weight 0, but their scales must not be NaN or infinite
            auto clear_rows = [&](int from, int to) {
                for (int j = lane; j < (to - from) * (kRowBytes / 16); j += 32)
                    reinterpret_cast<uint4 *>(vt + from * kRowBytes)[j] = make_uint4(0, 0, 0, 0);
                __syncwarp();
            };
            if (rows < 16 * kT) clear_rows(rows, 16 * kT);
            // Where a column ends inside the unit, the rows past its end are other columns': they stay. If one of them
            // has such a scale, the columns take turns, the longest first, and each clears what it does not see.
            unsigned on = (1u << n) - 1, left = 0;   // columns of the pass, columns of later passes
            int upto = rows, shortest = rows;
            auto rows_of = [&](int c) { return max(0, min(w.unit, min(row1, len[c]) - r0)); };
#pragma unroll
            for (int c = 0; c < kCols; c++)
                if (c < n) shortest = min(shortest, rows_of(c));
            bool apart = false;
            if (shortest < rows) {
                bool bad = false;
                for (int j = lane; j < (rows - shortest) * 8; j += 32) {
                    const unsigned char *const scale = vt + (shortest + (j >> 3)) * kRowBytes + (j & 7) * kQ8BlockBytes;
                    bad = bad || (*reinterpret_cast<const unsigned short *>(scale) & 0x7c00u) == 0x7c00u;
                }
                apart = __any_sync(0xffffffffu, bad);
                if (apart) left = on;
            }
            const unsigned *const vrow = reinterpret_cast<const unsigned *>(vt) + 2 * t * Row<false>::kPitch;
            auto value = [&](auto m) __attribute__((always_inline)) {
                constexpr int M = decltype(m)::value;
                VFrag f[kT];
#pragma unroll
                for (int j = 0; j < kT; j++) load_v<M, false>(vrow + j * 16 * Row<false>::kPitch, g, f[j]);
#pragma unroll
                for (int c = 0; c < kCols; c++) {
                    if (!(on >> c & 1)) continue;
                    float a[16];
#pragma unroll
                    for (int e = 0; e < 16; e++) a[e] = 0.0f;
                    if (i > 0) {
                        tmem_ld16(tmem + 128 * c + 16 * M, a);
                        tmem_wait_ld();
                    }
                    float ae[2][4], ao[2][4];
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        ae[e >> 2][e & 3] = a[e];
                        ao[e >> 2][e & 3] = a[8 + e];
                    }
#pragma unroll
                    for (int j = 0; j < kT; j++) add_values(f[j], ph[c][j], pl[c][j], ae, ao);
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        a[e] = ae[e >> 2][e & 3];
                        a[8 + e] = ao[e >> 2][e & 3];
                    }
                    tmem_st16(tmem + 128 * c + 16 * M, a);
                }
            };
            for (;;) {
                if (apart) {
                    __syncwarp();
                    int c_at = 0, most = -1;
#pragma unroll
                    for (int c = 0; c < kCols; c++)
                        if ((left >> c & 1) && rows_of(c) > most) {
                            most = rows_of(c);
                            c_at = c;
                        }
                    clear_rows(most, upto);
                    upto = most;
                    on = 1u << c_at;
                    left &= ~on;
                }
                value(Int<0>{});
                value(Int<1>{});
                value(Int<2>{});
                value(Int<3>{});
                if (left == 0) break;
            }
            tmem_wait_st();
            __syncwarp();
            vp += step;
            if (lane == 0 && i + 1 < nw) {
                if (apart) fence_async_shared();   // generic writes to the slot come before the copy's
                fetch(i + 1, vp, 1);
            }
            phase ^= 1;
        };
        for (int i = 0; i < nw; i++) {
            const int rows = min(w.unit, row1 - (first + i * w.unit * kWarps));
            if (rows > 16)
                work(Int<2>{}, i, rows);
            else
                work(Int<1>{}, i, rows);
        }

        // ---- merge: the warps of the CTA, two columns at a time, then the cluster, then the runs
        const int items = group * 64;
        const bool one_run = w.runs == 1 && p.out != nullptr;
        float2 *const wml = reinterpret_cast<float2 *>(smem + C::kOffMl);
        auto cpart = [&](int c) { return reinterpret_cast<float4 *>(smem + C::kOffQ + c * C::kQBytes); };
        auto cml = [&](int c) { return reinterpret_cast<float2 *>(smem + C::kOffCml) + 8 * c; };
#pragma unroll
        for (int c0 = 0; c0 < kCols; c0 += 2) {
            if (c0 >= n) break;
#pragma unroll
            for (int c = c0; c < c0 + 2; c++) {
                if (c >= n) break;
                sum_rows(run[c]);
                float2 *const ml = wml + (c - c0) * 8 * kWarps;
                if (g == 0) {
                    ml[(2 * t) * kWarps + warp] = make_float2(run[c].m[0], run[c].l[0]);
                    ml[(2 * t + 1) * kWarps + warp] = make_float2(run[c].m[1], run[c].l[1]);
                }
                float a[4][16];
#pragma unroll
                for (int m = 0; m < 4; m++)
#pragma unroll
                    for (int e = 0; e < 16; e++) a[m][e] = 0.0f;
                if (nw > 0) {
#pragma unroll
                    for (int m = 0; m < 4; m++) tmem_ld16(tmem + 128 * c + 16 * m, a[m]);
                    tmem_wait_ld();
                }
                float acc[8][2][4];
#pragma unroll
                for (int m = 0; m < 4; m++)
#pragma unroll
                    for (int e = 0; e < 16; e++) acc[2 * m + (e >> 3)][(e >> 2) & 1][e & 3] = a[m][e];
                store_warp_partial<false>(reinterpret_cast<float *>(ring + (c - c0) * C::kPartial), acc, group, g, t);
            }
            __syncthreads();
#pragma unroll
            for (int c = c0; c < c0 + 2; c++)
                if (c < n)
                    fold_warps(smem + (c - c0) * C::kPartial, C::kRing, wml + (c - c0) * 8 * kWarps, items,
                               [&](int item, const Part &r) {
                                   cpart(c)[item] = r.a;
                                   if ((item & 63) == 0) cml(c)[item >> 6] = make_float2(r.m, r.l);
                               });
            if (c0 + 2 < n) __syncthreads();
        }
        cluster_sync_all();
        fold_cluster<kC, kCols>(cpart(0), cml(0), C::kQBytes / 16, n, items, rank, [&](int c, int item, const Part &r) {
            if (one_run) emit_item(p, base + c, kvh, group, item, r);
            const size_t row = (size_t)(kvh * group + (item >> 6)) * p.splits + w.run;
            reinterpret_cast<float4 *>(p.part_acc + (size_t)(base + c) * p.acc_slot + row * 256)[item & 63] = r.a;
            if (writes_pair<kC>(items, rank, item))
                *reinterpret_cast<float2 *>(p.part_ml + (size_t)(base + c) * p.ml_slot + row * 2) = make_float2(r.m, r.l);
        });
        cluster_arrive();   // no CTA may leave, or start over, while another still reads its partials
        if (p.out != nullptr && !one_run) {
            int *const ctr = g_arrive_cols + (size_t)p.arrive_region * kArriveRegionInts +
                             (size_t)(base * p.n_kv + kvh) * p.arrive_stride + rank;
            __syncthreads();
            if (tid == 0) {
                const int last = arrive_acq_rel(ctr) == w.runs - 1;
                if (last) *ctr = 0;
                s_last = last;
            }
            __syncthreads();
            if (s_last) {
                // as many columns at a time as fit the rings
                const int slice = (items / kC + 1) * w.runs * 16, fit = max(1, min(n, kWarps * C::kRing / slice));
                for (int c = 0; c < n; c += fit) {
                    const int m = min(fit, n - c);
                    // (the staged fold takes the runs in one order; clusters of four and eight join shares of them, as
                    // the single-column body does)
                    if (Split<kC>::kShare == 1 &&
                        fold_runs_staged<kC>(p, base + c, m, kvh, group, w.runs, rank, smem, kWarps * C::kRing, bar_fold,
                                             fold_phase, reinterpret_cast<float2(*)[kStagedRow]>(smem + C::kOffFold), landed))
                        fold_phase ^= 1;
                    else
                        fold_runs<kC, 1, 8>(p, base + c, m, kvh, group, w.runs, rank, nullptr);
                }
            }
        }
        cluster_wait();
        __syncthreads();
        if (lane == 0) fence_async_shared();   // partials were written over the rings; a next round's copies follow
        }   // a live run of these columns
        sh.group += sh.hop;   // the cluster's next group of columns
        if (sh.group >= groups) break;
        find_group(sh, p.n_slots, base, end);
        plan();
    }
    if (!landed && status) atomicCAS(status, 0, 21);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc<1>(s_tmem, kTmemCols);
    }
}

template <int kC>
int launch(cudaStream_t stream, DecodeParams p) {
    static std::mutex mu;
    static int *status_word[64] = {};   // nullptr: device not set up yet
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (status_word[dev] == nullptr) {
            const cudaError_t e =
                cudaFuncSetAttribute(attn_decode_cols<kC>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
            if (e != cudaSuccess) return (int)e;
            status_word[dev] = device_status_word();
            if (status_word[dev] == nullptr) return launch_status();
        }
    }
    // (up to kMaxCols in a launch: 40 columns of 100 rows took 115 us as grids of the single-column body)
    for (int left = p.n_slots; left > 0; left -= kMaxCols) {
        p.n_slots = min(left, kMaxCols);
        if (int e = launch_pdl(attn_decode_cols<kC>, dim3(p.n_kv * p.run_cap * kC), dim3(kThreads), (size_t)Cfg::kSmem, stream,
                               kC, p, status_word[dev]))
            return e;
        p.len += kMaxCols * p.len_stride;
        p.q += kMaxCols * p.q_slot;
        p.part_acc += kMaxCols * p.acc_slot;
        p.part_ml += kMaxCols * p.ml_slot;
        if (p.out) p.out += kMaxCols * p.out_slot;
    }
    return 0;
}

}  // namespace

int launch_decode_cols(cudaStream_t stream, const DecodeParams &p, int cluster) {
    return cluster == 8 ? launch<8>(stream, p) : cluster == 4 ? launch<4>(stream, p) : launch<2>(stream, p);
}

}  // namespace hipml
