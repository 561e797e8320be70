// Split-K flash-decode over the q8_0 / q4_0 cache, head_dim 256: the body whose warps work alone.
//
// CPU definition: crates/hipml-core/src/ops.rs:449-518. Kernels replaced: crates/hipml-kernels/
// kernels/attn_decode_kv_w.hip:92-285 and attn_decode_kv.hip:251-374,427-484.
//
// A warp takes 16 or 32 rows (keys) at a time through the whole of the attention of its KV head's query
// heads: scores, softmax, values, with its own copy ring, its own running maximum and its own
// accumulators. Nothing between the set-up of a CTA and the merge of its eight warps is shared, so
// the loop has no CTA barrier at all.
//   * Ring: a unit of rows of K, then the same rows of V (one linear run of the cache each, 8,704 B
//     for 32 rows of q8_0), one bulk copy per unit, completion on an mbarrier per slot. While one unit is
//     worked on the others (two of three slots) are in flight, 139 KB per SM.
//   * Scores: mma.sync m16n8k16, codes as the A operand (16 keys x 16 dims), query as an f16 high
//     and low part in two chained MMAs as the B operand (8 columns, the group's heads). A code
//     pair becomes an f16 pair with one byte permute: code + 128 under a zero high byte is the
//     f16 subnormal (code + 128) * 2^-24; the offset leaves through the MMA's C operand (-2^-17 *
//     sum of the query over the block), the 2^-24 with the exponent's FMA. The block scale
//     multiplies whole accumulator rows. The query fragments lie in shared memory in the order
//     the MMA wants them (8 KB per CTA; in registers they would cost 64 a thread).
//   * Softmax: a lane holds keys g, g + 8 of heads 2t, 2t + 1. The maximum moves only when a score
//     exceeds it (one vote per unit), then the
//     accumulators are rescaled. Sums stay per lane until the end.
//   * Values: the weights become the B operand (k = key, n = head) by a transposing move of
//     8 x 8 tiles, as an exact f16 high + low pair after multiplication with the block's scale; the
//     codes are the A operand (16 dims x 16 keys), converted exactly (0x6400 | (code + 128) is
//     1152 + code). 64 accumulators per lane hold all 256 dims x 8 heads.
// What bounds it: long caches the HBM stream and the issue rate together (100,000 rows: 42 - 45 us a
// layer in a row = 4.85 - 5.15 TB/s, 33 us of it in the loop; 1,555 warp instructions per 32 rows of K and V, where 64-row
// tiles with CTA barriers and softmax through shared memory took 2,370, 57 us a layer); short ones
// the chain of dependent latencies (8,192 rows: 10.0 us, before 16).
//
// Merge: the eight warps' partials through shared memory, then the CTAs of a cluster, each of which
// folds a slice of the outputs and is sent the others' share of it, then, where a head has more
// than one cluster, through memory: the last cluster to arrive at the slice's counter folds it.
// Every sum runs in a fixed order, so the result does not depend on who arrives last.
#include <atomic>
#include <mutex>

#include "decode_warp_body.cuh"

namespace hipml {

namespace {

using namespace warp_body;

// kWide: one CTA per SM with up to 255 registers a thread and units of up to 32 rows (a query fragment
// read from shared memory serves two tiles, four MMA chains run side by side). Otherwise two CTAs per
// SM with 128 registers and units of 16 rows: twice as many, smaller CTAs.
template <bool kQ4, bool kWide>
struct Cfg {
    static constexpr int kUnitRows = kWide ? 32 : 16;
    static constexpr int kRow = kQ4 ? kQ4RowBytes : kRowBytes;
    static constexpr int kSlot = kUnitRows * kRow;                 // 8704 / 4608, half of it when not wide
    static constexpr int kSlots = kQ4 ? 5 : 3;                     // odd (see release)
    static constexpr int kRing = kSlots * kSlot;                   // per warp; later the warp's partial (8 heads)
    static_assert(kRing >= 8 * kHeadPitch * 4, "a warp's partial fits its ring");
    static constexpr int kOffQ = kWarps * kRing;                   // query fragments [16 steps][32 lanes]
    static constexpr int kOffBias = kOffQ + 16 * 32 * 16;          // [8 blocks][4] {head 2t, 2t + 1, 2t, 2t + 1}
    static constexpr int kOffMl = kOffBias + 8 * 4 * 16;           // [8 heads][warps] {reference, sum}
    static constexpr int kOffRow = kOffMl + kWarps * 8 * 8;        // the row to append: K, V
    static constexpr int kOffBar = kOffRow + 2 * kRow;             // a warp's slots each, then the last fold's
    static constexpr int kOffInMl = kOffBar + kWarps * kSlots * 8 + 16;   // (two more: the last fold's, the inbox's)
    static constexpr int kOffIn = (kOffInMl + 8 * 8 * 8 + 15) / 16 * 16;  // partials of the cluster's CTAs (wide)
    static constexpr int kSmem = kWide ? kOffIn + 8 * 256 * 4 : kOffInMl;
    static_assert((kWide ? 1 : 2) * (kSmem + 512 + 1024) <= 228 * 1024, "CTAs per SM");
};

// Arrival counters of the fold inside the split pass (see decode_arrive_region).
__device__ int g_arrive_warps[kArriveRegions * kArriveRegionInts];

// Several slots sharing one round of CTAs (a one-dimensional grid): CTA b takes the b-th live run in
// (slot, head, run) order, found by a scan over the slots' run counts. s_len: the live lengths.
// Called by all threads; s_plan is free again after the next CTA barrier.
template <int kUnitRows>
__device__ __forceinline__ Work plan_slots(const DecodeParams &p, const int *s_len, int *s_plan) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        const int quota = shared_quota_warp(s_len, 1, 0, p.n_slots, p.splits, p.share_slots, p.n_kv);
        const int b = blockIdx.x;
        int base = 0;
        if (lane == 0) s_plan[0] = -1;
        __syncwarp();
        for (int s0 = 0; s0 < p.n_slots; s0 += 32) {
            const int s = s0 + lane;
            const int n = s < p.n_slots ? s_len[s] : 0;
            const int per = s < p.n_slots ? shared_runs_of((n + 63) >> 6, quota) : 0;
            const int runs = per * p.n_kv;
            int incl = runs;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            const int first = base + incl - runs;
            if (runs > 0 && b >= first && b < first + runs) {
                const int r = b - first;
                s_plan[0] = s;
                s_plan[1] = r / per;
                s_plan[2] = r - (r / per) * per;
                s_plan[3] = per;
                s_plan[4] = n;
            }
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    Work w;
    w.slot = s_plan[0];
    w.kvh = s_plan[1];
    w.run = s_plan[2];
    w.runs = s_plan[3];
    w.len = s_plan[4];
    w.row0 = w.row1 = 0;
    w.unit = kUnitRows;
    if (w.slot >= 0) {
        const int tiles = div_up(w.len, 16);
        w.row0 = min((int)((long long)w.run * tiles / w.runs) * 16, w.len);
        w.row1 = min((int)((long long)(w.run + 1) * tiles / w.runs) * 16, w.len);
        if (w.row1 - w.row0 <= 16 * kWarps) w.unit = 16;
    }
    return w;
}

// kC: CTAs per cluster, which share a run. One stream: grid (n_kv * runs * kC, slots); several slots
// sharing the device: a one-dimensional grid of its CTA slots (kC = 1).
template <bool kQ4, int kC, bool kWide>
__global__ void __launch_bounds__(kThreads, kWide ? 1 : 2) attn_decode_warps(DecodeParams p, int *status) {
    using C = Cfg<kQ4, kWide>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_plan[8];
    __shared__ int s_len[64];   // live lengths of the slots that share a plan
    griddep_launch();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int group = p.n_heads / p.n_kv;
    const int rank = kC > 1 ? (int)cluster_rank() : 0;
    unsigned char *const ring = smem + warp * C::kRing;
    const unsigned ring_addr = smem_u32(ring), bar = smem_u32(smem + C::kOffBar) + warp * C::kSlots * 8;
    const unsigned bar_fold = smem_u32(smem + C::kOffInMl) - 16, bar_in = bar_fold + 8;
    const int items = group * 64;
    static_assert(kC == 1 || kWide, "clusters are wide");
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < C::kSlots; i++) mbar_init(bar + 8 * i, 1);
        if (warp == 0) {
            mbar_init(bar_fold, 1);
            if (kC > 1) mbar_init(bar_in, 1);
        }
        mbar_init_fence();
        if (kC > 1 && warp == 0) mbar_arrive_expect_tx(bar_in, inbox_bytes<kC>(items, rank));
    }
    if constexpr (kC > 1) cluster_arrive();   // (waited for before anything is sent to another CTA)
    uint4 *const qf = reinterpret_cast<uint4 *>(smem + C::kOffQ);
    const float4 *const bias = reinterpret_cast<const float4 *>(smem + C::kOffBias);
    bool landed = true;
    int off = 0;                 // the current unit's slot: its offset in the ring, its barrier and phase
    unsigned full = bar, phase = 0;

    // Before the grids ahead of this one are done, nothing they may write can be relied on: not the
    // cache rows, not the query, not even the live lengths. But the lengths as they stand are a good
    // guess (a step's layers share them), enough to plan with and to ask L2 for the first rows while
    // the grid ahead drains. Whatever comes of it is checked below.
    const bool shared_plan = kC == 1 && p.share_slots > 0;
    const int first_slot = shared_plan ? tid : (int)blockIdx.y;
    const bool reads_len = !shared_plan || tid < p.n_slots;
    const int *len_at = p.len + p.len_offset + first_slot * p.len_stride;
    auto read_len = [&]() { return live_len(p, __ldcg(len_at)); };
    Work w;
    if (shared_plan) {
        if (reads_len) s_len[tid] = read_len();
        __syncthreads();
        w = plan_slots<C::kUnitRows>(p, s_len, s_plan);
    } else {
        w = plan_stream<kC, C::kUnitRows>(p, first_slot, rank, read_len());
    }
    // This warp's units are rows row0 + unit * (warp + 8 i), i < nw. Only the last one can be short or
    // hold the row to append (the last live row).
    int nw, last_rows;
    unsigned unit_bytes, last_bytes, step;   // step: bytes from one unit of the warp to its next
    const unsigned char *kp, *vp;
    size_t head_byte;
    auto aim = [&]() {
        const int first = w.row0 + w.unit * warp;
        nw = first < w.row1 ? div_up(w.row1 - first, w.unit * kWarps) : 0;
        last_rows = min(w.unit, w.row1 - (first + w.unit * kWarps * (nw - 1)));
        unit_bytes = (unsigned)(w.unit * C::kRow);
        last_bytes = (unsigned)(last_rows * C::kRow);
        step = unit_bytes * kWarps;
        head_byte = (size_t)max(w.slot, 0) * p.kv_slot_bytes + (size_t)w.kvh * p.stride * C::kRow;
        kp = p.k + head_byte + (size_t)first * C::kRow;
        vp = p.v + head_byte + (size_t)first * C::kRow;
    };
    auto fetch = [&](int i, const unsigned char *src, unsigned dst, unsigned bar_full) {   // unit i: one lane
        const unsigned bytes = i == nw - 1 ? last_bytes : unit_bytes;
        mbar_arrive_expect_tx(bar_full, bytes);
        bulk_load(dst, src, bytes, bar_full);
    };
    auto fetch_first = [&](int from, int to) {   // of the warp's units K, V, K, ... into the slots in order
#pragma unroll
        for (int i = 0; i < C::kSlots; i++)
            if (i >= from && i < to && i < 2 * nw)
                fetch(i >> 1, ((i & 1) ? vp : kp) + (size_t)(i >> 1) * step, ring_addr + i * C::kSlot, bar + 8 * i);
    };
    aim();
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < kPrefetch; i++)
            if (i < nw) {
                const unsigned bytes = i == nw - 1 ? last_bytes : unit_bytes;
                prefetch_l2(kp + (size_t)i * step, bytes);
                prefetch_l2(vp + (size_t)i * step, bytes);
            }
        // and for the small inputs, whose trip to memory is on the path of every launch that finds them cold: the query
        // rows of the group, the row to append, the gate (a warp each)
        if (w.slot >= 0) {
            const size_t row = (size_t)w.slot * p.row_slot + (size_t)w.kvh * 256;
            const bool appends = p.k_row != nullptr && w.row1 == w.len;
            if (warp == 1) ask_l2(p.q + (size_t)w.slot * p.q_slot + (size_t)w.kvh * group * 256, 1024LL * group);
            if (warp == 2 && appends) ask_l2(p.k_row + row, 1024);
            if (warp == 3 && appends) ask_l2(p.v_row + row, 1024);
            if (warp == 4 && p.gate != nullptr && w.run == 0)
                ask_l2(p.gate + (size_t)w.slot * p.out_slot + (size_t)w.kvh * group * p.out_head_stride, 1024LL * group);
        }
    }
    griddep_wait();
    if constexpr (kC > 1) cluster_wait();
    for (;;) {
        // (the small loads first: behind the rows they would wait for all of them)
        const int real_len = reads_len ? read_len() : 0;
        float2 x[2][2];
        const float *const qh = p.q + (size_t)max(w.slot, 0) * p.q_slot + (size_t)(w.kvh * group + g) * 256;
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int d = kQ4 ? k_word_dim_q4(warp, t, 2 * i) + 16 * k : k_word_dim(warp, 4 * k + t, 2 * i);
                x[k][i] = make_float2(0.0f, 0.0f);
                if (g < group && w.slot >= 0) x[k][i] = *reinterpret_cast<const float2 *>(qh + d);
            }
        if (lane == 0) fetch_first(0, 1);
        // query fragments, warp b makes block b's
        store_query<kQ4>(x, p.scale_log2, warp, lane, qf, reinterpret_cast<float *>(smem + C::kOffBias));
        const bool guessed_wrong = reads_len && real_len != (shared_plan ? s_len[tid] : w.len);
        if (!__syncthreads_or(guessed_wrong)) break;
        // Rare: the lengths changed after they were first looked at. What was fetched lands, unused (its
        // slot's barrier starts over), and the CTA plans again.
        if (lane == 0) {
            if (nw > 0) {
                for (unsigned spin = 0; !mbar_try_wait(full, phase) && spin < kSpinLimit; spin++) {}
                mbar_inval(full);
                mbar_init(full, 1);
            }
            mbar_init_fence();
        }
        if (shared_plan) {
            if (reads_len) s_len[tid] = real_len;
            __syncthreads();
            w = plan_slots<C::kUnitRows>(p, s_len, s_plan);
        } else {
            w = plan_stream<kC, C::kUnitRows>(p, w.slot, rank, real_len);
        }
        aim();
    }
    if (w.slot < 0) return;
    if (lane == 0) fetch_first(1, C::kSlots);
    float *const part_acc = p.part_acc + (size_t)w.slot * p.acc_slot + (size_t)w.kvh * group * p.splits * 256;
    float *const part_ml = p.part_ml + (size_t)w.slot * p.ml_slot + (size_t)w.kvh * group * p.splits * 2;
    // Partial slots without rows hold a neutral partial (zero sum, -inf maximum): those of the launched runs and the first
    // kNeutralSlots of the others that the caller has. The runs without rows write them, which have nothing else to do
    // (written by the live ones ahead of their first unit they were 1.2 of the 7.4 us of a layer of 672 rows, whose one
    // run has 31 empty slots beside it); the live ones only where there are no others.
    // (a wide CTA alone shares the device with other slots, and has no such runs)
    if constexpr (kC > 1 || !kWide) {
        auto neutral = [&](int run) {
            const int at = rank * kThreads + tid;
            if (p.out != nullptr) {
                for (int i = at; i < items; i += kC * kThreads)
                    reinterpret_cast<float4 *>(part_acc + ((size_t)(i >> 6) * p.splits + run) * 256)[i & 63] =
                        make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else {   // (scratch on any 4-byte boundary)
                for (int i = at; i < group * 256; i += kC * kThreads)
                    part_acc[((size_t)(i >> 8) * p.splits + run) * 256 + (i & 255)] = 0.0f;
            }
            if (rank == 0 && tid < group) {
                float *const ml = part_ml + ((size_t)tid * p.splits + run) * 2;
                ml[0] = -INFINITY;
                ml[1] = 0.0f;
            }
        };
        if (p.share_slots == 0 && !p.by_stride && p.run_cap > 0) {
            const int launched = min(p.splits, p.run_cap), idle = launched - w.runs;
            const int from = idle > 0 ? w.run : launched + w.run, hop = idle > 0 ? idle : launched;
            if (idle <= 0 || w.run >= w.runs)
                for (int r = from; r < max(launched, min(p.splits, kNeutralSlots)); r += hop) neutral(r);
        }
        if (w.run >= w.runs) return;
    }

    // Fused append: the warp whose last unit holds the new row quantises it (with the encoder's own
    // arithmetic) while its first unit is on the way, stores it to the cache and keeps its bytes for the
    // units, which were copied as they were before this step.
    unsigned char *const new_rows = smem + C::kOffRow;   // K row, V row
    bool append = false;
    if (p.k_row != nullptr) {
        const int pos = __ldcg(p.len + w.slot * p.len_stride + p.len_offset - 1);
        append = nw > 0 && pos == w.len - 1 && w.row1 == w.len && (div_up(w.row1 - w.row0, w.unit) - 1) % kWarps == warp;
        // the fused form appends the last live row; anything else is the caller's error
        if (w.run == 0 && w.kvh == 0 && rank == 0 && tid == 0 && pos != w.len - 1 && status) atomicCAS(status, 0, 22);
        if (append) {
            const size_t at = (size_t)w.slot * p.row_slot + (size_t)w.kvh * 256 + lane * 8;
            const float4 ka = __ldg(reinterpret_cast<const float4 *>(p.k_row + at));
            const float4 kb = __ldg(reinterpret_cast<const float4 *>(p.k_row + at) + 1);
            const float4 va = __ldg(reinterpret_cast<const float4 *>(p.v_row + at));
            const float4 vb = __ldg(reinterpret_cast<const float4 *>(p.v_row + at) + 1);
            if constexpr (kQ4) {
                q4_put8(ka, kb, lane, new_rows);
                q4_put8(va, vb, lane, new_rows + C::kRow);
            } else {
                q8_put8(ka, kb, lane, new_rows);
                q8_put8(va, vb, lane, new_rows + C::kRow);
            }
            __syncwarp();
            const size_t to = head_byte + (size_t)pos * C::kRow;
            row_store(p.kw + to, new_rows, C::kRow, lane, 32);
            row_store(p.vw + to, new_rows + C::kRow, C::kRow, lane, 32);
        }
    }

    float acc[8][2][4];
#pragma unroll
    for (int b = 0; b < 8; b++)
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[b][i][c] = 0.0f;
    Running run;
    start(run);

    auto wait = [&]() {
        unsigned spin = 0;
        while (!mbar_try_wait(full, phase)) {
            if (++spin > kSpinLimit) {   // the copy never landed: flag it and carry on
                landed = false;
                break;
            }
        }
    };
    // Every lane has read the current unit: its slot takes unit `i` of the source, then the next slot.
    auto release = [&](bool wrote, int i, const unsigned char *src) {
        __syncwarp();
        if (i < nw && lane == 0) {
            if (wrote) fence_async_shared();   // generic writes to the slot come before the copy's
            fetch(i, src, ring_addr + off, full);
        }
        off += C::kSlot;
        full += 8;
        if (off == C::kRing) {
            off = 0;
            full = bar;
            phase ^= 1;
        }
    };
    auto put_row = [&](unsigned char *unit, const unsigned char *row) {   // the new row's bytes into the unit
        if (lane < C::kRow / 16)
            reinterpret_cast<uint4 *>(unit + (last_rows - 1) * C::kRow)[lane] = reinterpret_cast<const uint4 *>(row)[lane];
        __syncwarp();
    };
    // One unit of up to 16 * kT rows; `rows` of them live, `fresh`: the last one is the row to append.
    auto work = [&](auto tiles, int i, int rows, bool fresh) __attribute__((always_inline)) {
        constexpr int kT = decltype(tiles)::value;
        const bool plain = rows == 16 * kT && !fresh;
        // ---- scores
        wait();
        unsigned char *const kt = ring + off;
        if (fresh) put_row(kt, new_rows);
        float s[kT][4];
#pragma unroll
        for (int j = 0; j < kT; j++)
#pragma unroll
            for (int c = 0; c < 4; c++) s[j][c] = 0.0f;
        const unsigned *const krow = reinterpret_cast<const unsigned *>(kt) + g * Row<kQ4>::kPitch;
        auto score = [&](auto m) __attribute__((always_inline)) {
            KFrag<kT> f;
            load_k<decltype(m)::value, kQ4, kT>(krow, t, f);
            add_scores<decltype(m)::value, kT>(f, qf + lane, bias + t, s);
        };
        score(Int<0>{});
        score(Int<1>{});
        score(Int<2>{});
        score(Int<3>{});
        release(!plain, i + (C::kSlots - 1) / 2, vp + (size_t)((C::kSlots - 1) / 2) * step);
        __half2 ph[kT][2], pl[kT][2];
        float corr[2];
        const int rows_of[2] = {rows, rows};
        if (softmax<kT>(s, rows_of, g, run, ph, pl, corr)) {
#pragma unroll
            for (int b = 0; b < 8; b++)
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int c = 0; c < 4; c++) acc[b][j][c] *= corr[c & 1];
        }
        // ---- values
        wait();
        unsigned char *const vt = ring + off;
        if (!plain) {
            if (fresh) put_row(vt, new_rows + C::kRow);
            // stale rows have weight 0, but their scales must not be NaN or infinite
            for (int j = lane; j < (16 * kT - rows) * (C::kRow / 16); j += 32)
                reinterpret_cast<uint4 *>(vt + rows * C::kRow)[j] = make_uint4(0, 0, 0, 0);
            __syncwarp();
        }
        const unsigned *const vrow = reinterpret_cast<const unsigned *>(vt) + 2 * t * Row<kQ4>::kPitch;
        constexpr int kTilePitch = 16 * Row<kQ4>::kPitch;
        auto value = [&](auto m) __attribute__((always_inline)) {
            constexpr int M = decltype(m)::value;
#pragma unroll
            for (int j = 0; j < kT; j++) {
                VFrag f;
                load_v<M, kQ4>(vrow + j * kTilePitch, g, f);
                add_values(f, ph[j], pl[j], acc[2 * M], acc[2 * M + 1]);
            }
        };
        value(Int<0>{});
        value(Int<1>{});
        value(Int<2>{});
        value(Int<3>{});
        release(!plain, i + (C::kSlots + 1) / 2, kp + (size_t)((C::kSlots + 1) / 2) * step);
        kp += step;
        vp += step;
    };
    for (int i = 0; i < nw; i++) {
        const bool last = i == nw - 1;
        const int rows = last ? last_rows : w.unit;
        if (kWide && rows > 16)
            work(Int<kWide ? 2 : 1>{}, i, rows, last && append);
        else
            work(Int<1>{}, i, rows, last && append);
    }
    // ---- merge of the warps: their partials lie over the rings (every copy has been consumed)
    sum_rows(run);
    float2 *const wml = reinterpret_cast<float2 *>(smem + C::kOffMl);      // [8 heads][warp]
    if (g == 0) {
        wml[(2 * t) * kWarps + warp] = make_float2(run.m[0], run.l[0]);
        wml[(2 * t + 1) * kWarps + warp] = make_float2(run.m[1], run.l[1]);
    }
    store_warp_partial<kQ4>(reinterpret_cast<float *>(ring), acc, group, g, t);
    __syncthreads();
    const bool one_run = w.runs == 1 && p.out != nullptr && p.xch.phases == 0;
    // the run's partial of one item, and the output where there is no other run
    auto run_done = [&](int item, const Part &r) {
        if (one_run) emit_item(p, w.slot, w.kvh, group, item, r);
        const size_t row = (size_t)(item >> 6) * p.splits + w.run;
        float *const acc_at = part_acc + row * 256 + 4 * (item & 63), *const ml_at = part_ml + row * 2;
        const bool with_ml = writes_pair<kC>(items, rank, item);
        if (p.out != nullptr) {
            *reinterpret_cast<float4 *>(acc_at) = r.a;
            if (with_ml) *reinterpret_cast<float2 *>(ml_at) = make_float2(r.m, r.l);
        } else {   // partials that are folded by a launch of their own: scratch on any 4-byte boundary
            acc_at[0] = r.a.x;
            acc_at[1] = r.a.y;
            acc_at[2] = r.a.z;
            acc_at[3] = r.a.w;
            if (with_ml) {
                ml_at[0] = p.unit_weights ? r.m - kPScaleLog2 : r.m;
                ml_at[1] = r.l;
            }
        }
    };
    float4 *const inbox = reinterpret_cast<float4 *>(smem + C::kOffIn);
    float2 *const inbox_ml = reinterpret_cast<float2 *>(smem + C::kOffInMl);
    fold_warps(smem, C::kRing, wml, items, [&](int item, const Part &r) {
        if constexpr (kC > 1)
            send_item<kC>(inbox, inbox_ml, bar_in, items, rank, item, r);
        else
            run_done(item, r);
    });
    // ---- merge of the cluster: this CTA folds slice `rank` of the items
    if constexpr (kC > 1) {
        landed &= await_inbox(bar_in, 0);
        fold_inbox<kC>(inbox, inbox_ml, items, rank, run_done);
    }
    // ---- merge of the runs: the last to arrive at the slice's counter folds it
    if (p.out != nullptr && !one_run) {
        int *const ctr = g_arrive_warps + (size_t)p.arrive_region * kArriveRegionInts +
                         (size_t)(w.slot * p.n_kv + w.kvh) * p.arrive_stride;
        if (p.xch.phases == 0) {
            __syncthreads();
            if (tid == 0) {
                const int last = arrive_acq_rel(ctr + rank) == w.runs - 1;
                if (last) ctr[rank] = 0;
                s_plan[0] = last;
            }
            __syncthreads();
            if (s_plan[0]) {
                // (in a cluster a CTA has half a head group's items or less: ordinary loads, one trip for the runs of a
                // deep stream, are as fast for 17 runs, 137 us against 141 for 16 layers of 3,000 rows)
                if constexpr (kC > 1)
                    fold_runs<kC, 18>(p, w.slot, w.kvh, group, w.runs, rank, nullptr);
                else if (!fold_runs_staged(p, w.slot, w.kvh, group, w.runs, smem, kWarps * C::kRing, bar_fold,
                                           reinterpret_cast<float2(*)[kStagedRow]>(smem + C::kOffQ), landed))
                    fold_runs<kC, 8>(p, w.slot, w.kvh, group, w.runs, rank, nullptr);
            }
        } else {
            // the exchange wants whole heads in one CTA: the cluster arrives as one
            __threadfence();
            if constexpr (kC > 1) {
                cluster_sync_all();
            } else {
                __syncthreads();
            }
            if (rank == 0) {
                if (tid == 0) {
                    const int last = arrive_acq_rel(ctr) == w.runs - 1;
                    if (last) ctr[0] = 0;
                    s_plan[0] = last;
                }
                __syncthreads();
                if (s_plan[0]) {
                    float *const staged = reinterpret_cast<float *>(smem);
                    for (int r = 0; r < kC; r++) fold_runs<kC, 8>(p, w.slot, w.kvh, group, w.runs, r, staged);
                    __syncthreads();
                    FoldAcc f;
                    if (warp < group) {
                        const float2 ml = reinterpret_cast<const float2 *>(staged + 8 * 256)[warp];
                        constexpr float kInv = 1.0f / kPScale;
#pragma unroll
                        for (int i = 0; i < 8; i++) f.a[i] = staged[warp * 256 + lane * 8 + i] * kInv;
                        f.big = ml.x;
                        f.den = ml.y * kInv;
                    }
                    fold_finish(p, status, w.slot, w.kvh, group, f);
                }
            }
        }
    }
    if (!landed && status) atomicCAS(status, 0, 21);
}


// The fold of the runs as a launch of its own: the same arithmetic, bit for bit. Grid (n_kv * slices, slots), a CTA a
// slice of the outputs; with the exchange, which wants whole heads in one CTA, (n_kv, slots). kBatch: runs whose
// loads are issued together.
template <int kC, int kUnitRows, int kBatch>
__global__ void __launch_bounds__(kThreads) attn_decode_warps_fold(DecodeParams p, int *status) {
    __shared__ int s_quota;
    __shared__ int s_len[64];
    __shared__ __align__(16) float staged[8 * 256 + 16];
    griddep_launch();
    griddep_wait();
    const bool exchange = p.xch.phases != 0;
    const int slices = gridDim.x / p.n_kv, kvh = blockIdx.x / slices, slice = blockIdx.x - kvh * slices;
    const int slot = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = p.n_heads / p.n_kv;
    const int len = live_len(p, p.len[slot * p.len_stride + p.len_offset]);
    int runs = p.splits;
    if (p.share_slots > 0) {
        if (tid < p.n_slots) s_len[tid] = live_len(p, p.len[tid * p.len_stride + p.len_offset]);
        __syncthreads();
        if (warp == 0) {
            const int q = shared_quota_warp(s_len, 1, 0, p.n_slots, p.splits, p.share_slots, p.n_kv);
            if (lane == 0) s_quota = q;
        }
        __syncthreads();
        runs = shared_runs_of((len + 63) >> 6, s_quota);
    } else if (!p.by_stride && p.run_cap > 0) {
        runs = balance(p, len, kC, kUnitRows).runs;
    }
    if (!exchange) {
        fold_runs<kC, kBatch>(p, slot, kvh, group, runs, slice, nullptr, slices);
        return;
    }
    for (int r = 0; r < kC; r++) fold_runs<kC, 8>(p, slot, kvh, group, runs, r, staged);
    __syncthreads();
    FoldAcc f;
    if (warp < group) {
        const float2 ml = reinterpret_cast<const float2 *>(staged + 8 * 256)[warp];
        constexpr float kInv = 1.0f / kPScale;
#pragma unroll
        for (int i = 0; i < 8; i++) f.a[i] = staged[warp * 256 + lane * 8 + i] * kInv;
        f.big = ml.x;
        f.den = ml.y * kInv;
    }
    fold_finish(p, status, slot, kvh, group, f);
}

}  // namespace

namespace {

// Clusters of the kernel that fit the device at once (cached per device; 0: none).
template <bool kQ4, int kC, bool kWide>
int setup(int *max_runs, int **status) {
    static std::mutex mu;
    static int *status_word[64] = {};   // nullptr: device not set up yet
    static int active[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    std::lock_guard<std::mutex> lock(mu);
    if (status_word[dev] == nullptr) {
        auto kernel = attn_decode_warps<kQ4, kC, kWide>;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<kQ4, kWide>::kSmem);
        if (e != cudaSuccess) return (int)e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kC * 64);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = Cfg<kQ4, kWide>::kSmem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kC;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
        if (e != cudaSuccess) return (int)e;
        active[dev] = n;
        status_word[dev] = device_status_word();
        if (status_word[dev] == nullptr) return launch_status();
    }
    *max_runs = active[dev];
    *status = status_word[dev];
    return 0;
}

template <bool kQ4, int kC, bool kWide>
int launch(cudaStream_t stream, const DecodeParams &p, int slots) {
    int active = 0, *status = nullptr;
    if (int e = setup<kQ4, kC, kWide>(&active, &status)) return e;
    // (run_cap and share_slots count two CTAs per SM)
    DecodeParams q = p;
    q.n_slots = slots;
    dim3 grid(q.n_kv * q.splits, slots);
    if (q.share_slots > 0) {
        if (kWide) q.share_slots /= 2;
        grid = dim3(q.share_slots, 1);
    } else if (!q.by_stride && q.run_cap > 0) {
        q.run_cap = max(1, min(q.run_cap / ((kWide ? 2 : 1) * kC), active / q.n_kv));
        grid = dim3(q.n_kv * min(q.splits, q.run_cap) * kC, slots);
    }
    bool second_launch = false;
    if (q.out != nullptr) {
        q.arrive_stride = kC;
        q.arrive_region = decode_arrive_region(stream, (long long)slots * q.n_kv * kC);
        if (q.arrive_region < 0) {
            second_launch = true;
            q.out = nullptr;
        }
    }
    // several columns over one cache: side by side (not with the tail of an exchange)
    const bool columns = !kQ4 && kC > 1 && kWide && slots > 1 && q.kv_slot_bytes == 0 && q.k_row == nullptr &&
                         q.xch.phases == 0;
    const int rc = columns ? launch_decode_cols(stream, q, kC)
                           : launch_pdl(attn_decode_warps<kQ4, kC, kWide>, grid, dim3(kThreads),
                                        (size_t)Cfg<kQ4, kWide>::kSmem, stream, kC, q, status);
    if (rc != 0 || !second_launch) return rc;
    q.out = p.out;
    // Slices while their CTAs are few (672 rows 16.4 us with the split pass in one, 10.0 in eight; 16 slots of up to 3,000
    // rows 24.3 in one, 26.4 in four); many loads at once where there can be many runs (one slot of 256: 39.8 us by
    // eights, 25.4; 64 slots of few: 16.4, 18.7).
    constexpr int kUnitRows = Cfg<kQ4, kWide>::kUnitRows;
    int slices = q.xch.phases ? 1 : (kC > 4 ? kC : 4);
    while (slices > 1 && slots * q.n_kv * slices > (kC > 1 ? 2 * device_sms() : 64)) slices /= 2;
    return launch_pdl(q.splits > 16 ? attn_decode_warps_fold<kC, kUnitRows, 18> : attn_decode_warps_fold<kC, kUnitRows, 8>,
                      dim3(q.n_kv * slices, slots), dim3(kThreads), 0, stream, 1, q, status);
}

template <int kC, bool kWide>
int launch_c(cudaStream_t stream, const DecodeParams &p, int slots) {
    return p.q4 ? launch<true, kC, kWide>(stream, p, slots) : launch<false, kC, kWide>(stream, p, slots);
}

}  // namespace

// Which form. One stream (or columns of one) has ~37 SMs per KV head: clusters of two, wide (8,192 rows: 11.5 us
// a layer while partials were still read, against 14.4 with two small CTAs per SM and 13.1 with clusters of four,
// of which only 33 fit the device); clusters of eight up to the 1,023 rows that the engine's policy gives fewer than
// 128 splits, where one holds a head and nothing is folded through memory (672 rows, launches in a row: 6.1 us, of four
// 7.8, of two 7.8), while the device holds those of two launches (15: with eight KV heads the next launch waits for
// this one, 11.3 us against 8.1 with pairs; with six, whose next launch finds room for one head in two, 7.3 against 7.8);
// of four up to 519 (300 rows: 6.2 us, of eight 6.6, of two 7.7; at 100 rows pairs are as quick, 6.2 against 6.1).
// Several slots: no clusters, a head has too few CTAs to pair them; wide up to 28 (slot, head) pairs (4 KV heads, 5
// slots of 512 .. 3,000 rows: 14.3 us a layer against 14.6, 7 of 512 .. 8,192: 21.7, 25.7), beyond that the twice as fine
// runs of the small CTAs balance better where the last fold is not the longer part (8 slots of 512 .. 8,192: 24.1 us
// against 24.4, 16: 39.8, 41.6; 10: 28.1, 27.4).
int launch_decode_warps(cudaStream_t stream, const DecodeParams &p, int slots) {
    const bool one_stream = !p.by_stride && p.run_cap >= 4 && p.share_slots == 0;
    if (one_stream)
        return p.splits >= 128 || p.run_cap < 16 || (p.splits > 64 && p.n_kv > 6) ? launch_c<2, true>(stream, p, slots)
               : p.splits > 64                                                    ? launch_c<8, true>(stream, p, slots)
                                                                                  : launch_c<4, true>(stream, p, slots);
    return p.share_slots > 0 && slots * p.n_kv <= 28 ? launch_c<1, true>(stream, p, slots)
                                                     : launch_c<1, false>(stream, p, slots);
}

}  // namespace hipml
