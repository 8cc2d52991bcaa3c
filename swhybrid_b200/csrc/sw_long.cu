// sw_long.cu -- first pass for long record pairs: the query passes of one
// pair run concurrently in the warps of one block.
//
// The reference splits its GPU work into an "inter-sequence" kernel (one
// record per thread, src/CUDAKernel.cu:63-192) and sends records of 6,144
// residues or more to its CPU re-calculation instead
// (src/CUDAWorker.cu:144-201).  On B200 a long pair in the bulk kernel is a
// long serial chain of column steps in one group, so a DB whose residues sit
// in few long records leaves most of the GPU idle at the end.  Here a pair
// longer than the cut-over is scored by a pipeline of P warps, one warp per
// query pass of 32 x R rows: warp w runs an anti-diagonal wavefront (lane t one
// column behind lane t-1) on pass w, D = 2K column steps behind warp w-1, and
// takes the H/F of its first row's upper neighbour from a shared-memory ring
// that warp w-1's last thread fills.  The warps stay in step through one block
// barrier every K column steps (no flag waits):
//   * warp w-1's last thread writes column c at pipeline step (w-1)D + c + 31
//     and warp w's first thread reads it a step ahead of its own, at wD + c - 1,
//     K steps later, so a barrier always separates the write from the read;
//   * the ring holds 128 >= 3K columns, so the entry is overwritten (column
//     c + 128) at least K steps after it was read, again across a barrier.
// The per-pair cost of the pipeline is (P-1)D + 31 steps of fill and drain
// against ncols >= cut-over steps of work.  A block holds G such pipelines
// (G x P warps) that share the query profile and claim pairs independently;
// a pipeline's pair starts and ends at a barrier.  Each block takes a whole
// SM (it requests the SM's shared memory), so the long pairs run on the SMs
// the concurrent bulk launch leaves free.
//
// Bound: the latency of a column step (a pair's steps are serial), then issue
// when several warps share a scheduler.  So a step has one instruction per row
// in its serial chain (forward_short), no branch and no bounds guard: columns
// outside the pair run on zero-score residues, which raise no score, and the
// profile words, the residue and the ring entry are read a step ahead.  A step
// measured 133 / 171 / 251 / 347 clocks at 4 / 8 / 16 / 24 rows with one warp per
// scheduler (183 / 187 / 280 / 374 with the columns' checks in every step).
// Between them, 6, 12 and 20 rows keep a pass's padding small (query 375 in one
// pass: 251 clocks at 16 rows, 220 at 12).  A record much longer than the others
// would still hold the launch for its columns times that: it is cut into windows
// (sw_windows) that are units of their own and merge by maximum.
// Query 1,900 against 20,200 records of which 200 hold 43 % of the residues:
// 17.5 ms before (two half-columns per thread, guarded steps, 3 warps of 24 rows
// per pair, pipelines crowded on few SMs), 5.5 now.
#include <cstdint>

#include <cuda_runtime.h>

#include "sw_device.cuh"
#include "sw_long.h"
#include "sw_wavefront.cuh"

namespace swb {

namespace {

constexpr int kLT = 32;                  // threads per pass (one warp)
constexpr int kLK = 32;                  // column steps between block barriers
constexpr int kLD = 2 * kLK;             // step lag of warp w behind warp w-1
constexpr int kLRing = 128;              // ring columns per link (>= 3K, power of 2)

// Threads per block the compiler plans registers for: as many warps as the
// register file holds at the row count's register need, without spills.
template <int R>
struct LongBlock {
    static constexpr int value = R <= 6 ? 768 : R <= 16 ? 512 : R <= 32 ? 384 : 256;
};

// One warp of a pipeline: query pass w of P against the pipeline's pair.
template <int R, class CELL>
struct LongWarp {
    static constexpr int T = kLT;
    static constexpr int NJ = (R + 7) / 8;
    static constexpr int SLOTS = GroupShape<T>::SLOTS;
    static constexpr int JSTRIDE = kCodes * SLOTS;
    const CELL& K;
    const int t;                          // lane
    const uint32_t HZ, FZ;
    const uint2* prof_p = nullptr;        // the pass's profile at this lane's slot
    uint2* ring_out = nullptr;            // link w -> w+1
    const uint2* ring_in = nullptr;       // link w-1 -> w
    bool ring_wr = false, ring_rd = false;
    uint32_t H[R], E[R];
    uint32_t S, out_h, out_f, prev_h;
    uint2 up;                             // lane 0: the row above, next column
    uint2 wa[NJ], wb[NJ];                 // this step's profile words
    uint32_t d;                           // the next step's residue pair
    const unsigned short* col = nullptr;
    int ncols = 0, c = 0;

    __device__ __forceinline__ explicit LongWarp(const CELL& cell)
        : K(cell), t((int)(threadIdx.x & 31)), HZ(cell.hz()), FZ(cell.fz()) {}

    // links: this pipeline's P - 1 rings of kLRing columns
    __device__ __forceinline__ void place(const uint2* prof, uint2* links, int w, int P) {
        prof_p = prof + (w * NJ) * JSTRIDE + t;
        ring_out = links + (size_t)(w + 1 < P ? w : 0) * kLRing;
        ring_in = links + (size_t)(w > 0 ? w - 1 : 0) * kLRing;
        ring_wr = t == T - 1 && w + 1 < P;
        ring_rd = w > 0;
    }
    __device__ __forceinline__ uint32_t residue(int i) const {
        return i >= 0 && i < ncols ? (uint32_t)__ldg(col + i) : kPadPair;
    }
    __device__ __forceinline__ void load(uint2 (&A)[NJ], uint2 (&B)[NJ], uint32_t pr) const {
        const uint2* const p0 = prof_p + (int)(pr & 0xffu) * SLOTS;
        const uint2* const p1 = prof_p + (int)((pr >> 8) & 0xffu) * SLOTS;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            A[j] = p0[j * JSTRIDE];
            B[j] = p1[j * JSTRIDE];
        }
    }
    // steps of a pass over a pair, in whole barrier intervals
    static __device__ __forceinline__ int span_of(int ncols) {
        return (ncols + T - 1 + kLK - 1) / kLK * kLK;
    }
    __device__ __forceinline__ void begin(const uint4* db, const Pair2& pr) {
        ncols = (int)pr.ncols;
        col = reinterpret_cast<const unsigned short*>(db) + (size_t)pr.off16 * 8;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            H[k] = HZ;
            E[k] = FZ;
        }
        S = HZ;
        out_h = HZ;
        out_f = FZ;
        prev_h = HZ;
        up = make_uint2(HZ, FZ);
        c = -t;
        load(wa, wb, residue(c));
        d = residue(c + 1);
    }
    // K column steps from step s0.  INSIDE: every lane's column and the two
    // loaded ahead lie inside the pair, and so does lane 0's next ring entry,
    // so nothing is checked.
    template <bool INSIDE>
    __device__ __forceinline__ void steps(int s0) {
        constexpr unsigned FULL = 0xffffffffu;
        if (!INSIDE && ring_rd && s0 == 0) up = ring_in[0];
#pragma unroll 2
        for (int s = s0; s < s0 + kLK; ++s) {
            uint32_t h_in = __shfl_up_sync(FULL, out_h, 1);
            uint32_t f_in = __shfl_up_sync(FULL, out_f, 1);
            h_in = t == 0 ? up.x : h_in;
            f_in = t == 0 ? up.y : f_in;
            // the row above for column s + 1; past the pair's end nothing
            // flows in (the link's entries there are not written)
            if (ring_rd) up = ring_in[(s + 1) & (kLRing - 1)];
            if (!INSIDE && s + 1 >= ncols) up = make_uint2(HZ, FZ);
            uint2 na[NJ], nb[NJ];
            load(na, nb, d);
            d = INSIDE ? (uint32_t)__ldg(col + c + 2) : residue(c + 2);
#pragma unroll
            for (int k = R - 1; k >= 0; --k)
                H[k] = K.diag_floor(k > 0 ? H[k > 0 ? k - 1 : 0] : prev_h,
                                    pack_k(k, wa[k / 8], wb[k / 8]), E[k]);
            uint32_t f = f_in;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                K.forward_short(H[k], E[k], f);
                if (k & 1) S = __vimax3_s16x2(S, H[k > 0 ? k - 1 : 0], H[k]);
            }
            out_h = H[R - 1];
            out_f = f;
            if (ring_wr && (INSIDE || c >= 0))
                ring_out[c & (kLRing - 1)] = make_uint2(out_h, out_f);
            prev_h = h_in;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                wa[j] = na[j];
                wb[j] = nb[j];
            }
            ++c;
        }
    }
    // the barrier interval that starts at this warp's step s0
    __device__ __forceinline__ void interval(int s0) {
        if (s0 >= T && s0 + kLK + 2 <= ncols) steps<true>(s0);
        else steps<false>(s0);
    }
    // the pass's maximum, in every lane
    __device__ __forceinline__ uint32_t maximum() const {
        uint32_t m = S;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            m = __vimax3_s16x2(m, __shfl_xor_sync(0xffffffffu, m, o), HZ);
        return m;
    }
};

// A finished pair's scores (lanes of m) at row + its sorted position; merge: a
// window's, by maximum (put_score's rule).
__device__ __forceinline__ void long_scores(int* scores, int row, int pos, int n_records, uint32_t m,
                                            int bias, int thresh, int* ovf_list, int* ovf_count,
                                            int ovf_cap, bool merge) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (pos + i >= n_records) break;
        const int s = i ? hi16(m) : lo16(m);
        int* const at = scores + row + pos + i;
        bool list = s >= thresh;
        if (!merge) *at = s - bias;
        else if (list) list = atomicMax(at, kListed) != kListed;
        else atomicMax(at, s - bias);
        if (list) {
            const int j = atomicAdd(ovf_count, 1);
            if (j < ovf_cap) ovf_list[j] = row + pos + i;
        }
    }
}

// Plain search: one query, units (windows, then pairs) claimed pipeline by
// pipeline.
template <int R, class CELL>
__global__ void __launch_bounds__(LongBlock<R>::value, 1) sw_long(const LongArgs a) {
    using W = LongWarp<R, CELL>;
    extern __shared__ uint2 smem[];
    __shared__ int s_next[kLongMaxWarps];                 // per pipeline: its next pair
    __shared__ uint32_t s_max[kLongMaxWarps];             // per warp: its pass's max
    const int P = a.passes;                               // warps per pipeline
    const CELL K(a.gap_oe, a.gap_e);
    build_profile<kLT, R>(smem, a.query, a.qlen, a.mat, P, K.profile_bias());
    const int warp = (int)(threadIdx.x >> 5);
    const int g = warp / P;                               // this warp's pipeline
    const int w = warp - g * P;                           // ... and its pass in it
    W x(K);
    x.place(smem, smem + (size_t)P * W::NJ * W::JSTRIDE + (size_t)g * (P > 1 ? P - 1 : 0) * kLRing, w,
            P);
    const bool leader = w == 0 && x.t == 0;
    int pair = 0, span = 0, total = 0, start = 0;
    bool active = false;
    // a pipeline's pair starts at a barrier (block step `at`, a multiple of K)
    // and lasts `total` steps, also a multiple of K
    auto begin_pair = [&](int v, int at) {
        pair = v;
        active = pair < a.count;
        if (active) {
            x.begin(a.db, pair < a.n_win ? a.win_pairs[pair]
                                         : a.pairs[a.pair_begin + pair - a.n_win]);
            span = W::span_of(x.ncols);
            total = (P - 1) * kLD + span;
            start = at;
        }
    };
    if (leader) s_next[g] = atomicAdd(a.counter, 1);
    __syncthreads();                                       // profile built, first claims made
    begin_pair(s_next[g], 0);
    for (int gs = 0;;) {                                   // block step
        const int s0 = gs - start - w * kLD;               // this warp's first step of the interval
        if (active && s0 >= 0 && s0 < span) x.interval(s0);    // warp-uniform, whole intervals
        gs += kLK;
        // barrier: pipelines whose pair ends here publish their passes' maxima
        // and (leader) claim the next pair; the OR says whether any pipeline
        // still has work after this barrier
        const bool ending = active && gs - start >= total;
        bool alive = active && !ending;
        uint32_t m = x.HZ;
        if (ending) {
            m = x.maximum();
            if (x.t == 0) s_max[warp] = m;
            if (leader) {
                const int v = atomicAdd(a.counter, 1);
                s_next[g] = v;
                alive = v < a.count;
            }
        }
        const int any = __syncthreads_or(alive ? 1 : 0);
        if (ending) {
            if (leader) {
                for (int i = 1; i < P; ++i) m = __vimax3_s16x2(m, s_max[warp + i], x.HZ);
                const bool win = pair < a.n_win;
                const int at = win ? (int)a.win_ids[pair] : a.pair_begin + pair - a.n_win;
                long_scores(a.scores, 0, 2 * at, a.n_records, m, (int)(x.HZ & 0xffffu),
                            a.ovf_thresh - K.stored_shift(), a.ovf_list, a.ovf_count, a.ovf_cap,
                            win);
            }
            begin_pair(s_next[g], gs);
        }
        if (!any) break;
    }
}

// One item of sw_long_items at R rows a lane (whole block).
template <int R, class CELL>
__device__ __forceinline__ void long_item(const LongItemArgs& a, const CELL& K, uint2* smem,
                                          uint32_t* s_max, const uint2 item, int qlen,
                                          bool new_query) {
    using W = LongWarp<R, CELL>;
    const int warp = (int)(threadIdx.x >> 5);
    const int query = (int)item.x;
    const int P = (qlen + 32 * R - 1) / (32 * R);
    const int G = kLongItemWarps / P;
    if (new_query)
        build_profile<kLT, R>(smem, a.queries + a.qoff[query], qlen, a.mat, P, K.profile_bias());
    const int g = warp / P, w = warp - g * P;
    const int pair = (int)item.y + g;
    const bool active = g < G && pair < a.n_pairs;
    W x(K);
    __syncthreads();                 // profile built
    int span = 0;
    if (active) {
        x.place(smem, smem + (size_t)P * W::NJ * W::JSTRIDE + (size_t)g * (P > 1 ? P - 1 : 0) * kLRing,
                w, P);
        x.begin(a.db, a.pairs[pair]);
        span = W::span_of(x.ncols);
    }
    // the item's first pair is its longest
    const int total = (P - 1) * kLD + W::span_of((int)a.pairs[item.y].ncols);
    for (int gs = 0; gs < total; gs += kLK) {
        const int s0 = gs - w * kLD;
        if (active && s0 >= 0 && s0 < span) x.interval(s0);
        __syncthreads();
    }
    uint32_t m = x.HZ;
    if (active) {
        m = x.maximum();
        if (x.t == 0) s_max[warp] = m;
    }
    __syncthreads();
    if (active && w == 0 && x.t == 0) {
        for (int i = 1; i < P; ++i) m = __vimax3_s16x2(m, s_max[warp + i], x.HZ);
        long_scores(a.scores, query * a.n_records, 2 * pair, a.n_records, m, (int)(x.HZ & 0xffffu),
                    a.ovf_thresh - K.stored_shift(), a.ovf_list, a.ovf_count, a.ovf_cap, false);
    }
}

// Batched search and serving: items of one query and as many neighbouring
// pairs as a block of kLongItemWarps warps holds pipelines for (similar
// lengths, the table being longest first), claimed longest first.  One launch
// takes the items of every row count: it has its SMs while the first paired
// launch leaves them free, and a launch queued behind another one of the side
// stream met the next paired launch's blocks there and waited for their end (64
// queries of 50..5,000 residues against 57,000 records, paired shape 16x48: 324
// ms with a launch per row count, 229 now; 8x64: 289, 225).
template <class CELL>
__global__ void __launch_bounds__(32 * kLongItemWarps, 1) sw_long_items(const LongItemArgs a) {
    extern __shared__ uint2 smem[];
    __shared__ int s_item;
    __shared__ uint32_t s_max[kLongItemWarps];
    const CELL K(a.gap_oe, a.gap_e);
    int query = -1;
    while (true) {
        __syncthreads();                 // the previous item is done
        if (threadIdx.x == 0) s_item = atomicAdd(a.counter, 1);
        __syncthreads();
        if (s_item >= a.n_items) break;
        const uint2 item = a.items[s_item];
        const int qlen = (int)a.qlens[item.x];
        const bool new_query = (int)item.x != query;
        query = (int)item.x;
        switch (long_item_rows(qlen)) {
            case 4: long_item<4>(a, K, smem, s_max, item, qlen, new_query); break;
            case 8: long_item<8>(a, K, smem, s_max, item, qlen, new_query); break;
            default: long_item<16>(a, K, smem, s_max, item, qlen, new_query); break;
        }
    }
}

template <int R>
size_t long_smem(int passes, int pipelines) {
    constexpr int NJ = (R + 7) / 8;
    return (size_t)passes * NJ * kCodes * GroupShape<kLT>::SLOTS * sizeof(uint2) +
           (size_t)pipelines * (passes > 1 ? passes - 1 : 0) * kLRing * sizeof(uint2);
}

template <int R>
constexpr LongKernel linst() {
    return LongKernel{R,
                      {(const void*)&sw_long<R, CellWide>, (const void*)&sw_long<R, CellNarrow<0, 0>>,
                       (const void*)&sw_long<R, CellNarrow<12, 2>>,
                       (const void*)&sw_long<R, CellNarrow<12, 1>>},
                      &long_smem<R>, LongBlock<R>::value};
}

const LongItemKernel kLongItems{
    {(const void*)&sw_long_items<CellWide>, (const void*)&sw_long_items<CellNarrow<0, 0>>,
     (const void*)&sw_long_items<CellNarrow<12, 2>>, (const void*)&sw_long_items<CellNarrow<12, 1>>}};

const LongKernel kLongTable[] = {
    linst<4>(),  linst<6>(),  linst<8>(),  linst<12>(), linst<16>(),
    linst<20>(), linst<24>(), linst<32>(), linst<64>(),
};

}  // namespace

const LongItemKernel& long_item_kernel() { return kLongItems; }

size_t long_item_smem(int qlen) {
    const int R = long_item_rows(qlen), P = (qlen + 32 * R - 1) / (32 * R), G = kLongItemWarps / P;
    return R == 4 ? long_smem<4>(P, G) : R == 8 ? long_smem<8>(P, G) : long_smem<16>(P, G);
}

const LongKernel* long_kernels(int* n) {
    *n = (int)(sizeof(kLongTable) / sizeof(kLongTable[0]));
    return kLongTable;
}

}  // namespace swb
