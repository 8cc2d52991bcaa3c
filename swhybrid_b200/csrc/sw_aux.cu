// sw_aux.cu -- exact 32-bit re-score of overflowed records, score finalisation
// and top-k selection.
//
// The reference re-scores int8-overflowed records on the host after all
// workers have finished (RecalcWorker::recalc_launch, src/RecalcWorker.cpp:
// 99-268, 16 int16 lanes, saturating at 65535).  Here the first pass is
// already 16-bit, and the few records whose 16-bit lane may have wrapped are
// re-scored on the device in plain int32, from the compacted list the first
// pass appended to.  With SW_FLAG_REFERENCE_CAP the result is then clamped to
// 65535, which is exactly what the reference reports.
#include <cstdint>
#include "sw_aux.h"
#include "sw_device.cuh"

namespace swb {

constexpr int kRsRows = 16;        // query rows per lane in the 32-bit pass

// One warp per overflowed record: the same anti-diagonal wavefront as the
// first pass (32 lanes x 16 rows per pass), int32 arithmetic, profile taken
// from a shared copy of the matrix.  The boundary row between query passes is
// the warp's own scratch row, so any two records (of the same or of
// different queries) can be re-scored concurrently.
__global__ void __launch_bounds__(64) sw_rescore32(const RescoreArgs a) {
    __shared__ int smat[32 * 32];
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) smat[i] = a.mat[i];
    __syncthreads();
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    uint2* pb = a.scratch + (size_t)warp * a.max_cols;
    const int count = min(*a.ovf_count, a.ovf_cap);
    for (int it = warp; it < count; it += nwarps) {
        const int entry = a.ovf_list[it];
        int pos = entry;
        const uint8_t* query = a.query;
        int qlen = a.qlen;
        if (a.qoff) {
            const int q = entry / a.n_records;
            pos = entry - q * a.n_records;
            query = a.queries + a.qoff[q];
            qlen = (int)a.qlens[q];
        }
        const Pair2 pr = a.pairs[pos >> 1];
        const int sel = pos & 1;
        const uint8_t* seq = reinterpret_cast<const uint8_t*>(a.db + pr.off16);
        const int ncols = (int)pr.ncols;
        const int rows_per_pass = 32 * kRsRows;
        const int P = (qlen + rows_per_pass - 1) / rows_per_pass;
        int S = 0;
        for (int pass = 0; pass < P; ++pass) {
            int qc[kRsRows], H[kRsRows], E[kRsRows];
#pragma unroll
            for (int k = 0; k < kRsRows; ++k) {
                const int row = pass * rows_per_pass + lane * kRsRows + k;
                qc[k] = (row < qlen) ? (int)(query[row] & 31) * 32 : kZeroCode * 32;
                H[k] = 0;
                E[k] = 0;
            }
            int out_h = 0, out_f = 0, prev_h = 0, myd = kZeroCode;
            for (int s = 0; s < ncols + 31; ++s) {
                int d_in = __shfl_up_sync(FULL, myd, 1);
                int h_in = __shfl_up_sync(FULL, out_h, 1);
                int f_in = __shfl_up_sync(FULL, out_f, 1);
                if (lane == 0) {
                    d_in = kZeroCode;
                    h_in = 0;
                    f_in = 0;
                    if (s < ncols) {
                        d_in = seq[2 * s + sel] & 31;
                        if (pass > 0) {
                            const uint2 b = pb[s];
                            h_in = (int)b.x;
                            f_in = (int)b.y;
                        }
                    }
                }
                __syncwarp();
                const int c = s - lane;
                if (c >= 0 && c < ncols) {
                    int diag = prev_h, f = f_in;
#pragma unroll
                    for (int k = 0; k < kRsRows; ++k) {
                        int h = max(diag + smat[qc[k] + d_in], E[k]);
                        h = max(max(h, f), 0);
                        diag = H[k];
                        H[k] = h;
                        S = max(S, h);
                        const int hq = h - a.gap_oe;
                        E[k] = max(E[k] - a.gap_e, hq);
                        f = max(f - a.gap_e, hq);
                    }
                    out_h = H[kRsRows - 1];
                    out_f = f;
                    if (lane == 31 && pass + 1 < P) pb[c] = make_uint2((uint32_t)out_h, (uint32_t)out_f);
                }
                prev_h = h_in;
                myd = d_in;
                __syncwarp();
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) S = max(S, __shfl_xor_sync(FULL, S, o));
        if (lane == 0) a.scores[entry] = S;
        __syncwarp();
    }
}

// Windows of long pairs, one block per pair (blockIdx.x < the number of pairs
// to cut).  A pair's columns are one serial chain in the first pass, so a DB
// whose longest pairs hold more columns than an evenly loaded group gets would
// end on them.  No alignment of the query that scores above 0 spans more than
// W columns (its gap costs stay below the sum of its best match scores), so
// every one lies inside one of a set of windows that overlap by at least
// W - 1 columns, and the record's score is the maximum over its windows.
// Each window gets a table entry and a copy of its columns of its own (and
// with it a boundary row of its own: rows are addressed by stream position),
// so the first pass scores it like any pair.  Bound by latency: a few MB
// copied and a prefix sum over the counts of the pairs before (n_w^2 / 2
// 8-byte loads in all, n_w in the hundreds).
__global__ void __launch_bounds__(kWindowThreads) sw_windows(const WindowArgs a) {
    __shared__ int s_sum;
    const int p = (int)blockIdx.x;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    int before = 0;
    for (int i = (int)threadIdx.x; i < p; i += kWindowThreads)
        before += window_count((int)a.pairs[i].ncols, a.len, a.stride);
    before = __reduce_add_sync(0xffffffffu, before);
    if ((threadIdx.x & 31) == 0 && before) atomicAdd(&s_sum, before);
    __syncthreads();
    const int first = s_sum;
    const Pair2 pr = a.pairs[p];
    const int n = (int)pr.ncols;
    const int count = window_count(n, a.len, a.stride), step = window_step(n, a.len, a.stride);
    const int units = a.len / 8;
    const uint4* const src = a.db + pr.off16;
    uint4* const dst = a.db + a.base + (size_t)first * units;
    for (int w = (int)threadIdx.x; w < count; w += kWindowThreads) {
        a.win_pairs[first + w] = Pair2{a.base + (uint32_t)(first + w) * (uint32_t)units,
                                       (uint32_t)max(min(a.len, n - w * step), 0)};
        a.win_ids[first + w] = (uint32_t)p;
    }
    const int src_units = (n + 7) / 8;
    for (int i = (int)threadIdx.x; i < count * units; i += kWindowThreads) {
        const int w = i / units, u = i - w * units;
        const int from = w * (step / 8) + u;
        if (from < src_units) dst[i] = src[from];
    }
}

// A warp's largest key, in every lane.
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long key) {
    const uint32_t hi = (uint32_t)(key >> 32);
    const uint32_t top = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t lo = __reduce_max_sync(0xffffffffu, hi == top ? (uint32_t)key : 0u);
    return ((unsigned long long)top << 32) | lo;
}

// Top-k, one block: the first k of 4096 64-bit keys, descending.  Key = score
// << 32 | ~record_index, so the order is score descending, then record index
// ascending.  In the first round the keys are made from the per-position
// scores (clamped when asked) and the position -> record permutation, and the
// record-order score array is filled.  Bound: latency.  Up to kTopkSelect
// hits the block takes its maximum k times (4 keys a thread in registers, two
// warp reductions and one barrier each, about 200 clocks); for more hits it
// finds the last one's key bit by bit (two warp reductions and a barrier a bit),
// and only the last round sorts the hits (k = 500 of 40,000 records, three
// rounds: 97 us when each sorted its 4,096 keys, 32 now).
__global__ void __launch_bounds__(kTopkThreads) sw_topk_round(const TopkArgs a) {
    __shared__ unsigned long long sk[kTopkThreads];
    constexpr int kPer = kTopkKeys / kTopkThreads;
    const long long base = (long long)blockIdx.x * kTopkKeys;
    const long long y = blockIdx.y;                 // query of a batch
    const long long ys = (a.rows && !a.keys_in) ? a.rows[y] : y;   // its score row
    unsigned long long* const out = a.keys_out + y * a.out_stride + (long long)blockIdx.x * a.k;
    if (a.count && threadIdx.x == 0) out[a.k] = (unsigned long long)(uint32_t)*a.count;
    unsigned long long mine[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const long long g = base + j * kTopkThreads + threadIdx.x;
        unsigned long long key = 0ull;
        if (g < a.n) {
            if (a.keys_in) {
                key = a.keys_in[y * a.in_stride + g];
            } else {
                int s = a.scores[ys * a.in_stride + g];
                if (a.cap && s > 65535) s = 65535;
                const uint32_t rec = a.perm[g];
                if (a.scores_by_record) a.scores_by_record[ys * a.rec_stride + rec] = s;
                if (s > 0) key = ((unsigned long long)(uint32_t)s << 32) | (0xffffffffu - rec);
            }
        }
        mine[j] = key;
    }
    if (a.k <= kTopkSelect) {
        const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
        static_assert(kTopkThreads == 1024, "one warp maximum per lane of the second reduction");
        unsigned long long best = 0ull;
#pragma unroll
        for (int j = 0; j < kPer; ++j) best = max(best, mine[j]);
        for (int i = 0; i < a.k; ++i) {
            const unsigned long long w = warp_max_key(best);
            unsigned long long* const s = sk + 32 * (i & 1);   // the other half is still read
            if (lane == 0) s[warp] = w;
            __syncthreads();
            const unsigned long long top = warp_max_key(s[lane]);
            if (threadIdx.x == 0) out[i] = top;
            if (best == top && top != 0ull) {      // keys differ: one thread holds it
                best = 0ull;
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    if (mine[j] == top) mine[j] = 0ull;
                    best = max(best, mine[j]);
                }
            }
        }
        return;
    }
    // The kk-th largest key bit by bit (keys differ, zeros aside): the keys of at
    // least T are the block's hits.
    static_assert(kTopkThreads == 1024 && kMaxTopK <= kTopkThreads, "one key per thread below");
    constexpr unsigned FULL = 0xffffffffu;
    const int t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
    __shared__ int s_count[2][32];
    __shared__ int s_place;
    int turn = 0;
    auto at_least = [&](unsigned long long key) {      // how many of the block's keys
        int c = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) c += mine[j] >= key;
        c = __reduce_add_sync(FULL, c);
        if (lane == 0) s_count[turn][warp] = c;
        __syncthreads();
        c = __reduce_add_sync(FULL, s_count[turn][lane]);
        turn ^= 1;                                     // the other half is still read
        return c;
    };
    // (only the bits in which the block's keys differ: a score's and a record's)
    unsigned long long any = 0ull, all = ~0ull;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        any |= mine[j];
        if (mine[j]) all &= mine[j];
    }
    auto warp_or = [&](unsigned long long v) {
        return (unsigned long long)__reduce_or_sync(FULL, (uint32_t)(v >> 32)) << 32 |
               __reduce_or_sync(FULL, (uint32_t)v);
    };
    any = warp_or(any);
    all = ~warp_or(~all);
    if (lane == 0) {
        sk[warp] = any;
        sk[32 + warp] = all;
    }
    if (t == 0) s_place = 0;
    int n_top = at_least(1ull);
    const int kk = min(a.k, n_top);
    any = warp_or(sk[lane]);
    all = ~warp_or(~sk[32 + lane]);
    __syncthreads();                     // sk is written again below
    unsigned long long T = n_top ? all : ~0ull;
    for (unsigned long long left = n_top ? any & ~all : 0ull; left && n_top > kk;) {
        const unsigned long long bit = 1ull << (63 - __clzll((long long)left));
        left ^= bit;
        const int c = at_least(T | bit);
        if (c >= kk) {
            T |= bit;
            n_top = c;
        }
    }
    const bool last = gridDim.x == 1;                  // only the last round's hits are sorted
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const bool hit = mine[j] >= max(T, 1ull);
        const unsigned hits = __ballot_sync(FULL, hit);
        int at = 0;
        if (lane == 0 && hits) at = atomicAdd(&s_place, __popc(hits));
        at = __shfl_sync(FULL, at, 0) + __popc(hits & ((1u << lane) - 1u));
        if (hit) (last ? sk : out)[at] = mine[j];
    }
    if (!last) {
        for (int i = kk + t; i < a.k; i += kTopkThreads) out[i] = 0ull;
        return;
    }
    __syncthreads();
    unsigned long long key = t < kk ? sk[t] : 0ull;
    for (int size = 2; size <= kTopkThreads; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            unsigned long long other;
            if (stride >= 32) {
                __syncthreads();                       // the step before has been read
                sk[t] = key;
                __syncthreads();
                other = sk[t ^ stride];
            } else {
                other = __shfl_xor_sync(FULL, key, stride);
            }
            key = ((t & size) == 0) == ((t & stride) == 0) ? max(key, other) : min(key, other);
        }
    if (t < a.k) out[t] = key;
}

}  // namespace swb
