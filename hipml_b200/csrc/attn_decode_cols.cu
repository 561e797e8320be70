// Split-K flash-decode of several columns of one q8_0 stream (a speculative draft's columns, head_dim 256):
// the body of attn_decode_warps.cu with the columns side by side. CPU definition per column:
// crates/hipml-core/src/ops.rs:449-518; launcher replaced: launch_kv::launch_cols_ptrs.
//
// The columns see the same rows but for the last few, so a warp loads and converts a unit's codes once and runs the
// MMAs of all of them on it. The heads of a group of columns are packed into tiles of eight, the MMA's eight result
// columns, up to four tiles: four columns of six heads take three (a column each took four: 512 of the tensor pipe's
// eight-cycle MMAs a unit, 8.6 us of scores, softmax and values for 8,192 rows), and five share a launch's CTAs. What
// does not fit the registers is the accumulators (64 a lane and tile): they live in tensor memory, 128 of its columns
// per tile, and come to the registers 16 at a time for the pair of blocks at hand (tcgen05.ld / st), so that the loops
// over these pairs can be loops: unrolled four times, as the single-column body with its accumulators in registers has
// them, their code came from beyond the SM's instruction cache in every launch (4 columns of 8,192 rows, with their
// append: 27.9 us a layer, rolled 24.6; of 32,768: 53.0 and 50.9).
//
// The cluster's and the runs' partials meet column after column, each run beginning with another column: so the CTAs
// that arrive last, and fold the runs of a column, are different ones. (One CTA with all four columns of 17 runs, 209 KB,
// took 8.4 us at the end of every launch.)
//
// Each column's arithmetic is that of its own launch, operation for operation -- the plan, the order of
// every sum, the movements of the references -- so its result is the same bits.
#include <mutex>

#include "decode_warp_body.cuh"

namespace hipml {

namespace {

using namespace warp_body;

constexpr int kTiles = 4;         // of eight heads, of the columns side by side
constexpr int kCols = 8;          // most columns side by side (of four heads or fewer)
constexpr int kUnitRows = 32;
constexpr unsigned kTmemCols = 512;
constexpr int kMaxCols = 32;      // of a launch
constexpr int kArriveBar = 1;     // named barriers of the columns' arrivals

struct Cfg {
    static constexpr int kSlot = kUnitRows * kRowBytes;
    static constexpr int kRing = 2 * kSlot;                        // per warp: a unit of K and one of V; later two partials
    static constexpr int kPartial = 8 * kHeadPitch * 4;
    static_assert(kRing >= 2 * kPartial, "a warp's partials fit its ring");
    static constexpr int kQBytes = 16 * 32 * 16;                   // a tile's query fragments, later its partial of the CTA
    static_assert(kQBytes == 8 * 1024, "eight heads of a partial");
    static constexpr int kBiasBytes = 8 * 4 * 16;
    static constexpr int kOffQ = kWarps * kRing;
    static constexpr int kOffBias = kOffQ + kTiles * kQBytes;
    static constexpr int kOffMl = kOffBias + kTiles * kBiasBytes;  // [heads][warps] {reference, sum}
    static constexpr int kOffCml = kOffMl + kTiles * kWarps * 8 * 8;   // the CTA's, per head
    static constexpr int kOffBar = kOffCml + kTiles * 8 * 8;
    static constexpr int kSmem = kOffBar + kWarps * 2 * 8;
    static_assert(kSmem + 1024 <= 227 * 1024, "one CTA per SM");
};

__device__ int g_arrive_cols[kArriveRegions * kArriveRegionInts];

// Which columns a cluster takes. Neighbouring columns with the same plan (the same units for every warp), at
// most `each` of them (as many as fit the tiles, in groups of one size), are a group; a cluster has run `run` of
// groups `group`, `group` + `hop`, ... Groups go to clusters of their own while a head has clusters to spare for
// their runs, and columns share conversions beyond (4 columns of 300 rows take 2 runs each: 8 clusters of the head's
// 18; of 8,192 rows 17: one cluster per run takes all four). `cap`: the clusters of a head; what its groups do not
// need ends at once, so there is one round of them and they take the groups in turn.
struct Share {
    int each, run, group, hop;
    unsigned starts;   // bit c: column c's plan is not column c - 1's
};
template <int kC>
__device__ __forceinline__ Share share_columns(const DecodeParams &p, int cap, int in_head, int group, const int *len) {
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
    const int most = min(kCols, 8 * kTiles / group);
    s.each = div_up(p.n_slots, max(side, div_up(p.n_slots, most)));
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
    __shared__ int s_last[kCols];
    __shared__ unsigned s_tmem;
    __shared__ int s_len[kMaxCols];
    griddep_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int group = p.n_heads / p.n_kv;
    const int rank = (int)cluster_rank();
    unsigned char *const ring = smem + warp * C::kRing;
    const unsigned ring_addr = smem_u32(ring), bar = smem_u32(smem + C::kOffBar) + warp * 16;
    if (lane == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 1);
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
    Share sh = share_columns<kC>(p, cap, in_head, group, s_len);
    int base, end;
    int groups = find_group(sh, p.n_slots, base, end);
    int n, first, row1, nw;
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
        for (int c = 0; c < n; c++) longest = max(longest, s_len[base + c]);
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
    if (lane == 0 && warp < n)
        ask_l2(p.q + (size_t)(base + warp) * p.q_slot + (size_t)kvh * group * 256, 1024LL * group);
    griddep_wait();
    unsigned phase = 0;
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
        // Head f of the group's columns is head f % group of column f / group. Query fragments of every tile, warp b
        // makes block b's (as in the single-column body).
        const int heads = n * group, tiles = div_up(heads, 8);
        float2 x[kTiles][2][2];
#pragma unroll
        for (int a = 0; a < kTiles; a++) {
            const int f = 8 * a + g, c = f / group;
            const float *const qh = p.q + (size_t)(base + c) * p.q_slot + (size_t)(kvh * group + f - c * group) * 256;
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    x[a][k][i] = make_float2(0.0f, 0.0f);
                    if (f < heads) x[a][k][i] = *reinterpret_cast<const float2 *>(qh + k_word_dim(warp, 4 * k + t, 2 * i));
                }
        }
        if (lane == 0 && nw > 0) {
            fetch(0, kp, 0);
            fetch(0, vp, 1);
        }
        auto query_of = [&](int a) { return reinterpret_cast<uint4 *>(smem + C::kOffQ + a * C::kQBytes); };
        auto bias_of = [&](int a) { return reinterpret_cast<float *>(smem + C::kOffBias + a * C::kBiasBytes); };
#pragma unroll
        for (int a = 0; a < kTiles; a++)
            if (a < tiles) store_query<false>(x[a], p.scale_log2, warp, lane, query_of(a), bias_of(a));
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
            sh = share_columns<kC>(p, cap, in_head, group, s_len);
            groups = find_group(sh, p.n_slots, base, end);
            plan();
            checked = true;
            continue;
        }
        checked = true;
        tc_fence_after();
        if (base >= p.n_slots) break;
        if (live) {   // a run of these columns that has rows
            // this warp's accumulators of tile a: lanes 32 * (warp % 4), columns 128 a + 64 * (warp / 4)
            const unsigned tmem = s_tmem + ((unsigned)(warp & 3) << 21) + 64u * (warp >> 2);
            // live rows of heads 2t, 2t + 1 of every tile (heads past the last: the longest's)
            int len[kTiles][2];
#pragma unroll
            for (int a = 0; a < kTiles; a++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int f = 8 * a + 2 * t + h;
                    len[a][h] = f < heads ? s_len[base + f / group] : row1;
                }

            Running run[kTiles];
#pragma unroll
            for (int a = 0; a < kTiles; a++) start(run[a]);
            auto work = [&](auto row_tiles, int i, int rows) __attribute__((always_inline)) {
                constexpr int kT = decltype(row_tiles)::value;
                const int r0 = first + i * w.unit * kWarps;
                // ---- scores of all tiles
                wait(0);
                float s[kTiles][kT][4];
#pragma unroll
                for (int a = 0; a < kTiles; a++)
#pragma unroll
                    for (int j = 0; j < kT; j++)
#pragma unroll
                        for (int e = 0; e < 4; e++) s[a][j][e] = 0.0f;
                const unsigned *const krow = reinterpret_cast<const unsigned *>(ring) + g * Row<false>::kPitch;
#pragma unroll 1
                for (int M = 0; M < 4; M++) {   // pairs of blocks
                    KFrag<kT> f;
                    load_k<0, false, kT>(krow + M * Row<false>::kPair, t, f);
#pragma unroll
                    for (int a = 0; a < kTiles; a++)
                        if (a < tiles)
                            add_scores<0, kT>(f, query_of(a) + lane + 4 * 32 * M,
                                              reinterpret_cast<const float4 *>(bias_of(a)) + t + 8 * M, s[a]);
                }
                __syncwarp();
                kp += step;
                if (lane == 0 && i + 1 < nw) fetch(i + 1, kp, 0);
                // ---- softmax (where the unit begins past a column's end, that column gets nothing from it)
                __half2 ph[kTiles][kT][2], pl[kTiles][kT][2];
                auto sight = [&](int a, int h) { return min(w.unit, min(row1, len[a][h]) - r0); };
                // Heads (a bit each) whose references move: all of a column as soon as one of them is exceeded, no others, as
                // in the column's own launch.
                unsigned moving = 0;
#pragma unroll
                for (int a = 0; a < kTiles; a++) {
                    if (a >= tiles) break;
                    const int rows_of[2] = {sight(a, 0), sight(a, 1)};
                    float nm[2], x[kT][4];
                    bool over[2];
                    exponents<kT, true>(s[a], rows_of, g, run[a], nm, x, over);
                    // (lane t of each group of four has heads 2t, 2t + 1)
                    if (over[0]) moving |= 1u << (8 * a + 2 * t);
                    if (over[1]) moving |= 2u << (8 * a + 2 * t);
                }
                if (__any_sync(0xffffffffu, moving != 0)) {
                    moving = __reduce_or_sync(0xffffffffu, moving);
                    const unsigned one = (1u << group) - 1;
                    for (int c = 0; c < n; c++)
                        if (moving >> (c * group) & one) moving |= one << (c * group);
                }
#pragma unroll
                for (int a = 0; a < kTiles; a++) {
                    if (a >= tiles) break;
                    const int rows_of[2] = {sight(a, 0), sight(a, 1)};
                    const unsigned mine = moving >> (8 * a);
                    auto decide = [&](const bool (&)[2], bool (&move)[2]) {
                        move[0] = mine >> (2 * t) & 1;
                        move[1] = mine >> (2 * t + 1) & 1;
                        return (mine & 0xff) != 0;
                    };
                    float corr[2];
                    if (softmax<kT, true>(s[a], rows_of, g, run[a], ph[a], pl[a], corr, decide) && i > 0) {
#pragma unroll 1
                        for (int b = 0; b < 4; b++) {
                            float v[16];
                            tmem_ld16(tmem + 128 * a + 16 * b, v);
#pragma unroll
                            for (int e = 0; e < 16; e++) v[e] *= corr[e & 1];
                            tmem_st16(tmem + 128 * a + 16 * b, v);
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
                auto rows_of = [&](int c) { return max(0, min(w.unit, min(row1, s_len[base + c]) - r0)); };
                int shortest = rows;
                for (int c = 0; c < n; c++) shortest = min(shortest, rows_of(c));
                bool apart = false;
                if (shortest < rows) {
                    bool bad = false;
                    for (int j = lane; j < (rows - shortest) * 8; j += 32) {
                        const unsigned char *const scale = vt + (shortest + (j >> 3)) * kRowBytes + (j & 7) * kQ8BlockBytes;
                        bad = bad || (*reinterpret_cast<const unsigned short *>(scale) & 0x7c00u) == 0x7c00u;
                    }
                    apart = __any_sync(0xffffffffu, bad);
                }
                const unsigned *const vrow = reinterpret_cast<const unsigned *>(vt) + 2 * t * Row<false>::kPitch;
                // the values of the unit for all heads, or for those of column `only` (begun: there is something to add to)
                auto value = [&](int M, auto masked, int only, bool begun) __attribute__((always_inline)) {
                    constexpr bool kMasked = decltype(masked)::value != 0;
                    VFrag f[kT];
#pragma unroll
                    for (int j = 0; j < kT; j++)
                        load_v<0, false>(vrow + M * Row<false>::kPair + j * 16 * Row<false>::kPitch, g, f[j]);
#pragma unroll
                    for (int a = 0; a < kTiles; a++) {
                        if (a >= tiles) break;
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; e++) v[e] = 0.0f;
                        if (begun) tmem_ld16(tmem + 128 * a + 16 * M, v);
                        float ve[2][4], vo[2][4];
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            ve[e >> 2][e & 3] = v[e];
                            vo[e >> 2][e & 3] = v[8 + e];
                        }
                        const bool keep = !kMasked || (8 * a + g) / group == only;
#pragma unroll
                        for (int j = 0; j < kT; j++) add_values<kMasked>(f[j], ph[a][j], pl[a][j], ve, vo, keep);
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            v[e] = ve[e >> 2][e & 3];
                            v[8 + e] = vo[e >> 2][e & 3];
                        }
                        tmem_st16(tmem + 128 * a + 16 * M, v);
                    }
                };
                if (!apart) {
#pragma unroll 1
                    for (int M = 0; M < 4; M++) value(M, Int<0>{}, 0, i > 0);
                } else {
                    int upto = rows;
                    unsigned left = (1u << n) - 1;
                    for (bool begun = i > 0; left != 0; begun = true) {
                        int c_at = 0, most = -1;
                        for (int c = 0; c < n; c++)
                            if ((left >> c & 1) && rows_of(c) > most) {
                                most = rows_of(c);
                                c_at = c;
                            }
                        __syncwarp();
                        clear_rows(most, upto);
                        upto = most;
                        left &= ~(1u << c_at);
                        tmem_wait_st();   // what the turn before stored is loaded again
#pragma unroll 1
                        for (int M = 0; M < 4; M++) value(M, Int<1>{}, c_at, begun);
                    }
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

            // ---- merge: the warps of the CTA, two tiles at a time, then the cluster, then the runs
            const int items = group * 64;   // of a column
            const bool one_run = w.runs == 1 && p.out != nullptr;
            float2 *const wml = reinterpret_cast<float2 *>(smem + C::kOffMl);    // [heads][warps]
            float4 *const cpart = reinterpret_cast<float4 *>(smem + C::kOffQ);   // [heads][64]: over the query fragments
            float2 *const cml = reinterpret_cast<float2 *>(smem + C::kOffCml);   // [heads]
#pragma unroll
            for (int a = 0; a < kTiles; a++) {
                if (a >= tiles) break;
                sum_rows(run[a]);
                if (g == 0) {
                    wml[(8 * a + 2 * t) * kWarps + warp] = make_float2(run[a].m[0], run[a].l[0]);
                    wml[(8 * a + 2 * t + 1) * kWarps + warp] = make_float2(run[a].m[1], run[a].l[1]);
                }
            }
#pragma unroll 1
            for (int a0 = 0; a0 < tiles; a0 += 2) {
                const int a1 = min(a0 + 2, tiles);
#pragma unroll 1
                for (int a = a0; a < a1; a++) {
                    float v[64];
#pragma unroll
                    for (int e = 0; e < 64; e++) v[e] = 0.0f;
                    if (nw > 0) tmem_ld64(tmem + 128 * a, v);
                    float acc[8][2][4];
#pragma unroll
                    for (int e = 0; e < 64; e++) acc[e >> 3][(e >> 2) & 1][e & 3] = v[e];
                    store_warp_partial<false>(reinterpret_cast<float *>(ring + (a - a0) * C::kPartial), acc,
                                              min(8, heads - 8 * a), g, t);
                }
                __syncthreads();
#pragma unroll 1
                for (int a = a0; a < a1; a++)
                    fold_warps(smem + (a - a0) * C::kPartial, C::kRing, wml + 8 * a * kWarps, min(8, heads - 8 * a) * 64,
                               [&](int item, const Part &r) {
                                   cpart[a * 512 + item] = r.a;
                                   if ((item & 63) == 0) cml[a * 8 + (item >> 6)] = make_float2(r.m, r.l);
                               });
                if (a1 < tiles) __syncthreads();
            }
            cluster_sync_all();
            // Column after column, beginning with another one in every run. Warps 0 .. group - 1 fold the cluster's partials
            // of a column; another one (the s-th itself where there is none) announces the run.
            auto column = [&](int s) { return (s + w.run) % n; };
            const bool meet = p.out != nullptr && !one_run;
            for (int s = 0; s < n; s++) {
                const int c = column(s), announcer = group < 8 ? group + s % (8 - group) : s;
                if (warp < group)
                    fold_cluster<kC>(cpart + c * items, cml + c * group, items, rank, [&](int item, const Part &r) {
                        if (one_run) emit_item(p, base + c, kvh, group, item, r);
                        const size_t row = (size_t)(kvh * group + (item >> 6)) * p.splits + w.run;
                        reinterpret_cast<float4 *>(p.part_acc + (size_t)(base + c) * p.acc_slot + row * 256)[item & 63] = r.a;
                        if (writes_pair<kC>(items, rank, item))
                            *reinterpret_cast<float2 *>(p.part_ml + (size_t)(base + c) * p.ml_slot + row * 2) =
                                make_float2(r.m, r.l);
                    });
                if (!meet) continue;
                const int threads = 32 * (group < 8 ? group + 1 : 8);
                if (warp == announcer) {
                    named_sync(kArriveBar + s, threads);
                    if (lane == 0) {
                        int *const ctr = g_arrive_cols + (size_t)p.arrive_region * kArriveRegionInts +
                                         (size_t)((base + c) * p.n_kv + kvh) * p.arrive_stride + rank;
                        const int last = arrive_acq_rel(ctr) == w.runs - 1;
                        if (last) *ctr = 0;
                        s_last[s] = last;
                    }
                    __syncwarp();
                } else if (warp < group) {
                    named_arrive(kArriveBar + s, threads);
                }
            }
            cluster_arrive();   // no CTA may leave, or start over, while another still reads its partials
            if (meet) {
                __syncthreads();
                for (int s = 0; s < n; s++)
                    if (s_last[s]) {
                        if constexpr (kC == 2)
                            fold_runs<kC, 18>(p, base + column(s), kvh, group, w.runs, rank, nullptr);
                        else
                            fold_runs<kC, 8>(p, base + column(s), kvh, group, w.runs, rank, nullptr);
                    }
            }
            cluster_wait();
            __syncthreads();
            if (lane == 0) fence_async_shared();   // partials were written over the rings; a next round's copies follow
        }
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
