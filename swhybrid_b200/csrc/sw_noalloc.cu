// sw_noalloc.cu -- scoring entry point that allocates no memory.
//
// Some callers cannot call cudaMalloc where they score: a request path that
// must never allocate once it has started (an allocation can block on the
// driver and stall every request queued behind it), or a plug-in living in a
// host process whose device memory is all reserved by that process's own
// allocator.  sw_score_noalloc serves them: the caller passes device inputs
// and a device output, and every byte of scratch the kernel needs comes from
// one file-scope __device__ array that is part of the loaded library image.
// That array (256 warps x 8192 columns x 8 bytes plus a 256-byte header,
// about 16 MiB) is held by every GPU that loads the library until the
// process exits.
//
// One warp scores one record as an anti-diagonal wavefront in int32: lane t
// holds R query rows, one column behind lane t-1.  R is the smallest compiled
// row count whose 32 R rows hold the query (4..64), so queries up to 2,048
// residues run in one pass with no boundary row, and as many warps as fit; a
// longer query runs in passes of 2,048 rows that hand their last row on
// through the warp's slice of the static array (as many warps as there are
// slices of the longest record's length).
//
// Bound: the ALU pipe (64 lanes per clock and SM): 4.5 instructions per cell
// (the maxima of H before F, of H, E and F, and half a vimax3 for the running
// one), 5.5 with the byte profile's extraction.  The profile is read from shared memory,
// one conflict-free 16- or 4-byte word per 4 rows; looking each cell up in the
// matrix cost a bank-conflicted load per cell.  10,000 records, query 375:
// 4,400 us a call before (256 warps, 512-row passes, matrix lookups), 527 now.
//
// A record is a serial chain of columns, so records longer than an even share
// of the columns are cut into windows that overlap by the longest span an
// alignment can have (see sw_windows in sw_aux.cu); their scores merge by
// atomicMax.  Work is claimed through counters in the static array: first the
// long records' windows, then the other records.
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <iterator>
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/swb200.h"

namespace {

constexpr int kNaSlices = 256;         // boundary rows of kNaMaxLen in the scratch
constexpr int kNaMaxLen = 8192;        // longest DB record accepted, in residues
constexpr int kNaHeader = 32;          // uint2 words before the boundary rows (256 B)
constexpr size_t kRowWords = (size_t)kNaSlices * kNaMaxLen;
constexpr size_t kScratchWords = (size_t)kNaHeader + kRowWords;
constexpr int kNaThreads = 256;
constexpr int kNaLookupThreads = 64;
constexpr int kNaCodes = 25;           // 0..23 and the zero-score code 24

// The header's fields, then one boundary row of (H, F) entries per warp.  Host
// code must not use this name as an address.
struct NaHeader {
    unsigned int record;       // records claimed by the sweep over the short ones
    unsigned int max_len;      // longest record (up to kNaMaxLen)
    unsigned long long item;   // items claimed by the sweep over the long ones
    unsigned long long error;  // a record longer than kNaMaxLen was skipped
    unsigned long long best;   // sum of the query rows' best scores
};
static_assert(sizeof(NaHeader) <= kNaHeader * sizeof(uint2), "header");
static __device__ __align__(256) uint2 g_noalloc_scratch[kScratchWords];

struct NaArgs {
    const uint8_t* query;
    int qlen;
    const uint8_t* residues;
    const uint64_t* offsets;
    int n;
    int gap_oe;
    int gap_e;
    int cap;
    uint2* scratch;          // device address of g_noalloc_scratch
    int32_t* scores;         // zero before
    int8_t row_best[32];     // per query code: its best score (at least 0)
    int8_t mat[1024];
};

// Length of record i; kNaMaxLen + 1 for anything longer.
__device__ __forceinline__ int na_len(const NaArgs& a, int i) {
    const uint64_t b = a.offsets[i], e = a.offsets[i + 1];
    return (e <= b) ? 0 : (e - b > (uint64_t)kNaMaxLen) ? kNaMaxLen + 1 : (int)(e - b);
}

// The header's max_len and best: what the windows are planned from.
__global__ void __launch_bounds__(kNaThreads) sw_noalloc_prepare(const NaArgs a) {
    NaHeader* h = reinterpret_cast<NaHeader*>(a.scratch);
    const int first = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const int step = (int)(gridDim.x * blockDim.x);
    int longest = 0;
    for (int64_t i = first; i < a.n; i += step) {
        const int len = na_len(a, (int)i);
        if (len <= kNaMaxLen) longest = max(longest, len);
    }
    long long best = 0;
    for (int i = first; i < a.qlen; i += step) best += a.row_best[a.query[i] & 31];
    longest = __reduce_max_sync(0xffffffffu, longest);
    if ((threadIdx.x & 31) == 0 && longest > 0) atomicMax(&h->max_len, (unsigned)longest);
    if (best > 0) atomicAdd(&h->best, (unsigned long long)best);
}

// Profile words of 4 rows: int32 scores, or signed bytes.
template <bool BYTES>
struct NaWord {
    using type = int4;
    static __device__ __forceinline__ int get(const int4& w, int i) {
        return i == 0 ? w.x : i == 1 ? w.y : i == 2 ? w.z : w.w;
    }
    static __device__ __forceinline__ int4 make(const int* v) {
        return make_int4(v[0], v[1], v[2], v[3]);
    }
};
template <>
struct NaWord<true> {
    using type = uint32_t;
    static __device__ __forceinline__ int get(uint32_t w, int i) {
        return (int)(int8_t)(w >> (8 * i));
    }
    static __device__ __forceinline__ uint32_t make(const int* v) {
        return (v[0] & 0xff) | (v[1] & 0xff) << 8 | (v[2] & 0xff) << 16 | (uint32_t)v[3] << 24;
    }
};

template <int R, bool BYTES>
size_t na_smem(int qlen) {
    const int passes = (qlen + 32 * R - 1) / (32 * R);
    return (size_t)passes * (R / 4) * kNaCodes * 32 * sizeof(typename NaWord<BYTES>::type);
}

// One record (or window) against the whole query: the warp's best score.
// PASSES: the query takes more than one pass (a step of a single pass has no
// branch: it is mostly latency).
template <int R, bool BYTES, bool PASSES, class WORD>
__device__ __forceinline__ int na_score(const NaArgs& a, const WORD* prof, int P, uint2* pb,
                                        const uint8_t* seq, int len) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NJ = R / 4, JSTRIDE = kNaCodes * 32;
    const int lane = (int)(threadIdx.x & 31);
    int S = 0;
    for (int pass = 0; pass < (PASSES ? P : 1); ++pass) {
        const WORD* const pp = prof + pass * NJ * JSTRIDE + lane;
        const bool rd = PASSES && pass > 0 && lane == 0;
        const bool wr = PASSES && pass + 1 < P && lane == 31;
        int H[R], E[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            H[k] = 0;
            E[k] = 0;
        }
        int out_h = 0, out_f = 0, prev_h = 0;
        int c = -lane;
        auto residue = [&](int i) {
            return (i >= 0 && i < len) ? (unsigned)__ldg(seq + i) : 24u;
        };
        // codes 25..31 (none is documented) score 0 like 24
        auto words_of = [&](unsigned code) { return pp + min(code & 31u, 24u) * 32; };
        // the profile words of this step's column and the next column's
        // residue are loaded a step ahead
        WORD w[NJ];
        {
            const WORD* const pd = words_of(residue(c));
#pragma unroll
            for (int j = 0; j < NJ; ++j) w[j] = pd[j * JSTRIDE];
        }
        unsigned d = residue(c + 1);
        uint2 row = make_uint2(0u, 0u);
        if (rd && len > 0) row = pb[0];
        // a column outside the record runs on zero-score residues: before it
        // all cells stay at 0, after it no score can rise
        for (int s = 0; s < len + 31; ++s, ++c) {
            if (PASSES) __syncwarp();    // orders the boundary row's stores and loads
            int h_in = __shfl_up_sync(FULL, out_h, 1);
            int f_in = __shfl_up_sync(FULL, out_f, 1);
            h_in = lane == 0 ? (PASSES ? (int)row.x : 0) : h_in;
            f_in = lane == 0 ? (PASSES ? (int)row.y : 0) : f_in;
            if (PASSES && rd) row = (c + 1 < len) ? pb[c + 1] : make_uint2(0u, 0u);
            WORD wn[NJ];
            const WORD* const pd = words_of(d);
#pragma unroll
            for (int j = 0; j < NJ; ++j) wn[j] = pd[j * JSTRIDE];
            d = residue(c + 2);
#pragma unroll
            for (int k = R - 1; k >= 0; --k)
                H[k] = __vimax3_s32((k > 0 ? H[k > 0 ? k - 1 : 0] : prev_h) +
                                        NaWord<BYTES>::get(w[k / 4], k % 4),
                                    E[k], 0);
            // F of the next row from max(H before F, 0): a later row's F never
            // gains from an H that F itself made (extending is no dearer than
            // opening), which leaves one add and one maximum per row in the
            // serial chain
            int f = f_in;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int t = H[k];
                const int h = max(t, f);
                H[k] = h;
                f = max(f - a.gap_e, t - a.gap_oe);
                E[k] = max(E[k] - a.gap_e, h - a.gap_oe);
                if (k & 1) S = __vimax3_s32(S, H[k > 0 ? k - 1 : 0], h);
            }
            out_h = H[R - 1];
            out_f = f;
            if (PASSES && wr && c >= 0 && c < len) pb[c] = make_uint2((uint32_t)out_h, (uint32_t)out_f);
            prev_h = h_in;
#pragma unroll
            for (int j = 0; j < NJ; ++j) w[j] = wn[j];
        }
        if (PASSES) __syncwarp();
    }
    return __reduce_max_sync(FULL, S);
}

template <int R, bool BYTES, int THREADS, int MIN_BLOCKS>
__global__ void __launch_bounds__(THREADS, MIN_BLOCKS) sw_score_noalloc_kernel(const NaArgs a) {
    using WORD = typename NaWord<BYTES>::type;
    extern __shared__ int4 na_prof[];
    WORD* const prof = reinterpret_cast<WORD*>(na_prof);
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NJ = R / 4;
    NaHeader* const h = reinterpret_cast<NaHeader*>(a.scratch);
    const int P = (a.qlen + 32 * R - 1) / (32 * R);
    for (int idx = (int)threadIdx.x; idx < P * NJ * kNaCodes * 32; idx += THREADS) {
        const int t = idx & 31;
        int rest = idx >> 5;
        const int d = rest % kNaCodes;
        rest /= kNaCodes;
        const int row0 = (rest / NJ * 32 + t) * R + rest % NJ * 4;
        int v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = row0 + i < a.qlen ? a.mat[(a.query[row0 + i] & 31) * 32 + d] : 0;
        prof[idx] = NaWord<BYTES>::make(v);
    }
    __syncthreads();
    const int lane = (int)(threadIdx.x & 31);
    const int warp = (int)((blockIdx.x * THREADS + threadIdx.x) >> 5);
    const long long warps = (long long)gridDim.x * (THREADS / 32);
    // windows: long enough that the overlap costs at most two thirds, and at
    // least a warp's even share of the columns
    const long long max_len = h->max_len;
    const long long share = (long long)((a.offsets[a.n] - a.offsets[0]) / (uint64_t)warps);
    long long span = 0, wlen = kNaMaxLen;
    if (a.gap_e > 0) {
        const long long over = (long long)h->best - 1 - (a.gap_oe - a.gap_e);
        span = a.qlen + (over > 0 ? over / a.gap_e : 0);
        const long long w = max(share, span + max(span / 2, 256ll));
        if (w + w / 4 < max_len) wlen = w;
    }
    const int L = (int)wlen, stride = (int)(L - span + 1);
    uint2* pb = a.scratch + kNaHeader;
    if (P > 1) {
        const long long row = max(min(max_len, wlen), 1ll);
        if (warp >= (long long)kRowWords / row) return;     // no boundary row left
        pb += warp * row;
    }
    auto score = [&](int rec, int start, int len, bool merge) {
        const uint8_t* seq = a.residues + a.offsets[rec] + start;
        int s = P > 1 ? na_score<R, BYTES, true>(a, prof, P, pb, seq, len)
                      : na_score<R, BYTES, false>(a, prof, P, pb, seq, len);
        if (lane == 0) {
            if (a.cap) s = min(s, 65535);
            if (merge) atomicMax(a.scores + rec, s);
            else a.scores[rec] = s;
        }
    };
    // The long records first, so that a unit claimed last is short.  An item
    // is window k of 4 neighbouring records, those of them that have one; of one
    // record where the claims are few (up to 16 a warp), since a warp scores an
    // item's records one after the other while others idle (us with 4 -> with 1:
    // 181 records, query 444 386 -> 196, 3,000 and 375 430 -> 288, 5,000 and
    // 1,500 2,047 -> 1,449).
    const int big = (int)min(max(share / 8, 128ll), (long long)L);
    if (big < max_len) {
        // (stride is only meaningful where a record is longer than a window)
        const long long windows = max_len <= L ? 1 : 1 + (max_len - L + stride - 1) / stride;
        const int per = a.n * windows > 16 * warps ? 4 : 1;
        const long long groups = ((long long)a.n + per - 1) / per;
        const long long items = groups * windows;
        while (true) {
            unsigned long long it = 0;
            if (lane == 0) it = atomicAdd(&h->item, 1ull);
            it = __shfl_sync(FULL, it, 0);
            if ((long long)it >= items) break;
            const int k = (int)((long long)it / groups);
            const long long rec = ((long long)it - k * groups) * per + (lane & (per - 1));
            const int len = rec < a.n ? na_len(a, (int)rec) : 0;
            const bool has = len > big && len <= kNaMaxLen &&
                             (k == 0 || (len > L && k <= (len - L + stride - 1) / stride));
            unsigned todo = __ballot_sync(FULL, has && lane < per);
            while (todo) {
                const int src = __ffs(todo) - 1;
                todo &= todo - 1;
                const int n = __shfl_sync(FULL, len, src);
                score((int)(rec - (lane & (per - 1))) + src, k > 0 ? k * stride : 0,
                      k > 0 ? min(L, n - k * stride) : min(L, n), n > L);
            }
        }
    }
    unsigned next = 0;
    if (lane == 0) next = atomicAdd(&h->record, 1u);
    while (true) {
        const unsigned rec = __shfl_sync(FULL, next, 0);
        if (rec >= (unsigned)a.n) break;
        if (lane == 0) next = atomicAdd(&h->record, 1u);
        const int len = na_len(a, (int)rec);
        if (len > kNaMaxLen) {
            if (lane == 0) atomicExch(&h->error, 1ull);
        } else if (len <= big) {
            score((int)rec, 0, len, false);
        }
    }
}

// Queries whose byte profile does not fit a block's shared memory (over 8,192
// residues, four passes of 51,200 bytes): passes of 512 rows, scores looked up in a shared copy of the
// matrix, one boundary row of kNaMaxLen per warp.
__global__ void __launch_bounds__(kNaLookupThreads) sw_score_noalloc_lookup(const NaArgs a) {
    constexpr int kRows = 16;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ int smat[1024];
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) smat[i] = a.mat[i];
    __syncthreads();
    NaHeader* const h = reinterpret_cast<NaHeader*>(a.scratch);
    const int lane = (int)(threadIdx.x & 31);
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    uint2* const pb = a.scratch + kNaHeader + (size_t)warp * kNaMaxLen;
    const int P = (a.qlen + 32 * kRows - 1) / (32 * kRows);
    while (true) {
        unsigned rec = 0;
        if (lane == 0) rec = atomicAdd(&h->record, 1u);
        rec = __shfl_sync(FULL, rec, 0);
        if (rec >= (unsigned)a.n) break;
        const int len = na_len(a, (int)rec);
        if (len > kNaMaxLen) {
            if (lane == 0) atomicExch(&h->error, 1ull);
            continue;
        }
        const uint8_t* seq = a.residues + a.offsets[rec];
        int S = 0;
        for (int pass = 0; pass < P; ++pass) {
            int qc[kRows], H[kRows], E[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int row = (pass * 32 + lane) * kRows + k;
                qc[k] = (row < a.qlen) ? (int)(a.query[row] & 31) * 32 : 24 * 32;
                H[k] = 0;
                E[k] = 0;
            }
            int out_h = 0, out_f = 0, prev_h = 0, myd = 24;
            for (int s = 0; s < len + 31; ++s) {
                int d_in = __shfl_up_sync(FULL, myd, 1);
                int h_in = __shfl_up_sync(FULL, out_h, 1);
                int f_in = __shfl_up_sync(FULL, out_f, 1);
                if (lane == 0) {
                    d_in = 24;
                    h_in = 0;
                    f_in = 0;
                    if (s < len) {
                        d_in = seq[s] & 31;
                        if (pass > 0) {
                            const uint2 v = pb[s];
                            h_in = (int)v.x;
                            f_in = (int)v.y;
                        }
                    }
                }
                __syncwarp();
                const int c = s - lane;
                if (c >= 0 && c < len) {
                    int diag = prev_h, f = f_in;
#pragma unroll
                    for (int k = 0; k < kRows; ++k) {
                        int hk = max(diag + smat[qc[k] + d_in], E[k]);
                        hk = max(max(hk, f), 0);
                        diag = H[k];
                        H[k] = hk;
                        S = max(S, hk);
                        const int hq = hk - a.gap_oe;
                        E[k] = max(E[k] - a.gap_e, hq);
                        f = max(f - a.gap_e, hq);
                    }
                    out_h = H[kRows - 1];
                    out_f = f;
                    if (lane == 31 && pass + 1 < P)
                        pb[c] = make_uint2((uint32_t)out_h, (uint32_t)out_f);
                }
                prev_h = h_in;
                myd = d_in;
                __syncwarp();
            }
        }
        S = __reduce_max_sync(FULL, S);
        if (lane == 0) a.scores[rec] = (a.cap && S > 65535) ? 65535 : S;
        __syncwarp();
    }
}

// The compiled row counts: one pass of 32 R rows up to 2,048 query residues.
struct NaKernel {
    int rows;
    int threads;             // per block
    int blocks;              // per SM
    const void* fn;
    size_t (*smem)(int qlen);
};
template <int R, bool BYTES, int THREADS, int MIN_BLOCKS>
constexpr NaKernel na_inst() {
    return NaKernel{32 * R, THREADS, MIN_BLOCKS,
                    (const void*)&sw_score_noalloc_kernel<R, BYTES, THREADS, MIN_BLOCKS>,
                    &na_smem<R, BYTES>};
}
// int32 profile words up to 512 rows (51 KB), bytes above.  One block per SM
// with as few warps as nearly fill its ALU pipe: a column step takes longer
// with every further warp on its scheduler, and the longest unit's columns are
// serial (12 rows, 10,000 records: 586 us with 8 warps, 648 with 12).
const NaKernel kNaKernels[] = {
    na_inst<4, false, 512, 1>(),  na_inst<8, false, 512, 1>(),
    na_inst<12, false, 256, 1>(), na_inst<16, false, 256, 1>(),
    na_inst<24, true, 256, 1>(),  na_inst<32, true, 256, 1>(),
    na_inst<48, true, 256, 1>(),  na_inst<64, true, 256, 1>(),
};

// What the first call on a device looks up.  It also loads every kernel a later
// call may take (the runtime otherwise loads each one when it is first used,
// which can allocate device memory and block) and allows it its shared memory.
struct NaDevice {
    void* scratch = nullptr;     // device address of the static array
    int sms = 0, max_smem = 0;
};
std::mutex g_na_mutex;
NaDevice g_na_device[64];

bool na_first_call(int device, NaDevice* d) {
    NaDevice x;
    if (cudaDeviceGetAttribute(&x.sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&x.max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) !=
            cudaSuccess ||
        cudaGetSymbolAddress(&x.scratch, g_noalloc_scratch) != cudaSuccess)
        return false;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, (const void*)sw_noalloc_prepare) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, (const void*)sw_score_noalloc_lookup) != cudaSuccess)
        return false;
    for (const NaKernel& k : kNaKernels)
        if (cudaFuncGetAttributes(&fa, k.fn) != cudaSuccess ||
            cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 x.max_smem - (int)fa.sharedSizeBytes) != cudaSuccess)
            return false;
    *d = x;
    return true;
}

}  // namespace

extern "C" sw_status sw_score_noalloc(int device, const sw_params* params, const uint8_t* d_query,
                                      uint32_t qlen, const uint8_t* d_residues,
                                      const uint64_t* d_offsets, uint32_t n_records,
                                      int32_t* d_scores, void* cuda_stream) {
    if (!params || (n_records && (!d_offsets || !d_scores)) || (qlen && !d_query) || device < 0 ||
        device >= 64)
        return SW_ERR_INVALID;
    if (params->gap_open < 0 || params->gap_extend < 0 ||
        params->gap_open + params->gap_extend > 1000)
        return SW_ERR_INVALID;
    for (int i = 0; i < 1024; ++i)
        if (params->matrix[i] < -127 || params->matrix[i] > 127) return SW_ERR_INVALID;
    if (qlen > (1u << 24) || n_records > (uint32_t)INT32_MAX) return SW_ERR_UNSUPPORTED;
    int prev = 0;
    if (cudaGetDevice(&prev) != cudaSuccess) return SW_ERR_CUDA;
    if (cudaSetDevice(device) != cudaSuccess) return SW_ERR_NO_DEVICE;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    sw_status rc = SW_OK;
    do {
        NaDevice dev;
        {
            std::lock_guard<std::mutex> lock(g_na_mutex);
            if (!g_na_device[device].scratch && !na_first_call(device, &g_na_device[device])) {
                cudaGetLastError();
                rc = SW_ERR_CUDA;
                break;
            }
            dev = g_na_device[device];
        }
        void* const addr = dev.scratch;
        if (n_records == 0) break;
        if (qlen == 0) {
            if (cudaMemsetAsync(d_scores, 0, (size_t)n_records * sizeof(int32_t), st) != cudaSuccess)
                rc = SW_ERR_CUDA;
            else if (cudaStreamSynchronize(st) != cudaSuccess)
                rc = SW_ERR_CUDA;
            break;
        }
        NaArgs a;
        a.query = d_query;
        a.qlen = (int)qlen;
        a.residues = d_residues;
        a.offsets = d_offsets;
        a.n = (int)n_records;
        a.gap_oe = params->gap_open + params->gap_extend;
        a.gap_e = params->gap_extend;
        a.cap = (params->flags & SW_FLAG_REFERENCE_CAP) ? 1 : 0;
        a.scratch = (uint2*)addr;
        a.scores = d_scores;
        for (int i = 0; i < 1024; ++i)
            a.mat[i] = (int8_t)(((i >> 5) >= 24 || (i & 31) >= 24) ? 0 : params->matrix[i]);
        for (int i = 0; i < 32; ++i) {
            a.row_best[i] = 0;
            for (int j = 0; j < 32; ++j) a.row_best[i] = std::max(a.row_best[i], a.mat[i * 32 + j]);
        }
        const NaKernel* k = nullptr;
        for (const NaKernel& x : kNaKernels)
            if (!k && (x.rows >= (int)qlen || &x == std::end(kNaKernels) - 1)) k = &x;
        const bool looked_up = k->smem((int)qlen) > (size_t)dev.max_smem;
        const void* fn = looked_up ? (const void*)&sw_score_noalloc_lookup : k->fn;
        const size_t smem = looked_up ? 0 : k->smem((int)qlen);
        const int threads = looked_up ? kNaLookupThreads : k->threads;
        // the header and the scores (merged by maximum) start at zero
        if (cudaMemsetAsync(addr, 0, sizeof(NaHeader), st) != cudaSuccess ||
            cudaMemsetAsync(d_scores, 0, (size_t)n_records * sizeof(int32_t), st) != cudaSuccess) {
            rc = SW_ERR_CUDA;
            break;
        }
        void* args[] = {&a};
        const unsigned prep = std::min<unsigned>(
            (unsigned)dev.sms, (std::max(n_records, qlen) + kNaThreads - 1) / kNaThreads);
        const unsigned grid =
            looked_up ? (unsigned)(kNaSlices / (kNaLookupThreads / 32))
                      : std::min<unsigned>((unsigned)(k->blocks * dev.sms), std::max(n_records, 1u));
        if (cudaLaunchKernel((const void*)sw_noalloc_prepare, dim3(prep), dim3(kNaThreads), args, 0,
                             st) != cudaSuccess ||
            cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, smem, st) != cudaSuccess) {
            cudaGetLastError();
            rc = SW_ERR_CUDA;
            break;
        }
        uint32_t err = 0;
        if (cudaMemcpyAsync(&err, (const char*)addr + offsetof(NaHeader, error), sizeof(err),
                            cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            rc = SW_ERR_CUDA;
            break;
        }
        if (err) rc = SW_ERR_UNSUPPORTED;
    } while (0);
    cudaSetDevice(prev);
    return rc;
}
