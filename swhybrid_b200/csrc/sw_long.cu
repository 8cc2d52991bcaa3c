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
// measured 134 / 176 / 265 / 352 clocks at 4 / 8 / 16 / 24 rows with one warp per
// scheduler (183 / 187 / 280 / 374 with the columns' checks in every step).
// Query 1,900 against 20,200 records of which 200 hold 43 % of the residues:
// 17.5 ms before (two half-columns per thread, guarded steps, 3 warps of 24 rows
// per pair, pipelines crowded on few SMs), 6.6 now.
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
    static constexpr int value = R <= 4 ? 768 : R <= 16 ? 512 : R <= 32 ? 384 : 256;
};

template <int R, class CELL>
__global__ void __launch_bounds__(LongBlock<R>::value, 1) sw_long(const LongArgs a) {
    constexpr int T = kLT;
    constexpr int NJ = (R + 7) / 8;
    constexpr int SLOTS = GroupShape<T>::SLOTS;
    constexpr int JSTRIDE = kCodes * SLOTS;
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ uint2 smem[];
    __shared__ int s_next[kLongMaxWarps];                 // per pipeline: its next pair
    __shared__ uint32_t s_max[kLongMaxWarps];             // per warp: its pass's max
    const int P = a.passes;                               // warps per pipeline
    const CELL K(a.gap_oe, a.gap_e);
    uint2* const prof = smem;
    uint2* const ring = smem + (size_t)P * NJ * JSTRIDE;  // G pipelines x (P-1) links
    build_profile<T, R>(prof, a.query, a.qlen, a.mat, P, K.profile_bias());
    const int warp = (int)(threadIdx.x >> 5);
    const int g = warp / P;                               // this warp's pipeline
    const int w = warp - g * P;                           // ... and its pass in it
    const int t = (int)(threadIdx.x & 31);
    const bool leader = (w == 0 && t == 0);
    const uint32_t HZ = K.hz(), FZ = K.fz();
    const int bias = (int)(HZ & 0xffffu);
    const int ovf_thresh = a.ovf_thresh - K.stored_shift();
    const uint2* const prof_p = prof + (w * NJ) * JSTRIDE + t;
    uint2* const links = ring + (size_t)g * (P > 1 ? P - 1 : 0) * kLRing;
    uint2* const ring_out = links + (size_t)(w + 1 < P ? w : 0) * kLRing;       // link w -> w+1
    const uint2* const ring_in = links + (size_t)(w > 0 ? w - 1 : 0) * kLRing;  // link w-1 -> w
    const bool ring_wr = t == T - 1 && w + 1 < P;
    const bool ring_rd = w > 0;
    uint32_t H[R], E[R];
    uint32_t S = HZ, out_h = HZ, out_f = FZ, prev_h = HZ;
    uint2 up = make_uint2(HZ, FZ);                        // lane 0: the row above, next column
    uint2 wa[NJ], wb[NJ];                                 // this step's profile words
    uint32_t d = kPadPair;                                // the next step's residue pair
    const unsigned short* col = reinterpret_cast<const unsigned short*>(a.db);
    int pair = 0, ncols = 0, span = 0, total = 0, start = 0, c = 0;
    bool active = false;
    auto residue = [&](int i) {
        return i >= 0 && i < ncols ? (uint32_t)__ldg(col + i) : kPadPair;
    };
    auto load = [&](uint2 (&A)[NJ], uint2 (&B)[NJ], uint32_t pr) {
        const uint2* const p0 = prof_p + (int)(pr & 0xffu) * SLOTS;
        const uint2* const p1 = prof_p + (int)((pr >> 8) & 0xffu) * SLOTS;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            A[j] = p0[j * JSTRIDE];
            B[j] = p1[j * JSTRIDE];
        }
    };
    // a pipeline's pair starts at a barrier (block step `at`, a multiple of K)
    // and lasts `total` steps, also a multiple of K
    auto begin_pair = [&](int v, int at) {
        pair = v;
        active = pair < a.pair_count;
        if (active) {
            const Pair2 pr = a.pairs[a.pair_begin + pair];
            ncols = (int)pr.ncols;
            span = (ncols + T - 1 + kLK - 1) / kLK * kLK;
            total = (P - 1) * kLD + span;
            start = at;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                H[k] = HZ;
                E[k] = FZ;
            }
            S = HZ;
            out_h = HZ;
            out_f = FZ;
            prev_h = HZ;
            col = reinterpret_cast<const unsigned short*>(a.db) + (size_t)pr.off16 * 8;
            c = -t;
            load(wa, wb, residue(c));
            d = residue(c + 1);
            up = make_uint2(HZ, FZ);
        }
    };
    if (leader) s_next[g] = atomicAdd(a.counter, 1);
    __syncthreads();                                       // profile built, first claims made
    begin_pair(s_next[g], 0);
    // K column steps of this warp from its step s0.  INSIDE: every lane's
    // column and the two loaded ahead lie inside the pair, and so does lane 0's
    // next ring entry, so nothing is checked.
    auto interval = [&](auto inside, int s0) {
        constexpr bool INSIDE = decltype(inside)::value;
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
    };
    for (int gs = 0;;) {                                   // block step
        const int s0 = gs - start - w * kLD;               // this warp's first step of the interval
        if (active && s0 >= 0 && s0 < span) {              // warp-uniform, whole intervals
            if (ring_rd && s0 == 0) up = ring_in[0];
            if (s0 >= T && s0 + kLK + 2 <= ncols) interval(Flag<true>{}, s0);
            else interval(Flag<false>{}, s0);
        }
        gs += kLK;
        // barrier: pipelines whose pair ends here publish their passes' maxima
        // and (leader) claim the next pair; the OR says whether any pipeline
        // still has work after this barrier
        const bool ending = active && gs - start >= total;
        bool alive = active && !ending;
        if (ending) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                S = __vimax3_s16x2(S, __shfl_xor_sync(FULL, S, o), HZ);
            if (t == 0) s_max[warp] = S;
            if (leader) {
                const int v = atomicAdd(a.counter, 1);
                s_next[g] = v;
                alive = v < a.pair_count;
            }
        }
        const int any = __syncthreads_or(alive ? 1 : 0);
        if (ending) {
            if (leader) {
                for (int i = 1; i < P; ++i) S = __vimax3_s16x2(S, s_max[warp + i], HZ);
                const int pos = 2 * (a.pair_begin + pair);
                const int s0 = lo16(S), s1 = hi16(S);
                a.scores[pos] = s0 - bias;
                if (s0 >= ovf_thresh) {
                    const int j = atomicAdd(a.ovf_count, 1);
                    if (j < a.ovf_cap) a.ovf_list[j] = pos;
                }
                if (pos + 1 < a.n_records) {
                    a.scores[pos + 1] = s1 - bias;
                    if (s1 >= ovf_thresh) {
                        const int j = atomicAdd(a.ovf_count, 1);
                        if (j < a.ovf_cap) a.ovf_list[j] = pos + 1;
                    }
                }
            }
            begin_pair(s_next[g], gs);
        }
        if (!any) break;
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

const LongKernel kLongTable[] = {
    linst<4>(), linst<8>(), linst<16>(), linst<24>(), linst<32>(), linst<64>(),
};

}  // namespace

const LongKernel* long_kernels(int* n) {
    *n = (int)(sizeof(kLongTable) / sizeof(kLongTable[0]));
    return kLongTable;
}

}  // namespace swb
