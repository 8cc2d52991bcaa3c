// sw_traceback.cu -- alignments (coordinates and CIGAR) of chosen DB records.
//
// The reference reports scores and record titles only (WorkerPool::showResult,
// src/WorkerPool.cpp:130-155); it has no traceback.  sw_traceback gives the
// caller the best local alignment of the query against each record it names
// (typically the top-k hits of a search):
//   * one block per record runs the exact int32 Gotoh recurrence: each warp is
//     an anti-diagonal wavefront over 128 query rows (32 lanes x 4), the warps
//     follow one another down the query and hand their last row on through
//     shared-memory rings (as the long-pair first pass does), and every cell's
//     4 direction bits are stored: H is not the diagonal's, H is not E, the next
//     E extends, the next F extends;
//   * the end cell is the first cell with the maximal H in column-major order
//     (record position, then query position);
//   * one warp then walks the bits back from the end cell: in H it stops at
//     H = 0 (it carries H along) and otherwise prefers the diagonal, then E,
//     then F; inside a gap it prefers "opened here" over "extended" on ties.  The 32 lanes look at the
//     next 32 cells along the diagonal (or along the gap), so a run of matches
//     costs one load per 32 cells.
// Bound: latency.  A 1,000 x 1,000 alignment is 1,250 column steps, each a chain
// of two shuffles and two instructions per row (F takes max(H before F, 0));
// each bit is the sign of a difference shifted into the word, and a step has no
// branch: columns outside the record run on zero-score residues.  The walk is a
// chain of loads, one per run.  Ten alignments of 1,000 x 1,000: 2,340 us a call before (one
// warp per record, 16 rows a lane in two passes, matrix lookups per cell, one
// dependent load per walked cell), 481 now.
// The direction bits take qlen x record length / 2 bytes per record, in a
// scratch buffer the context keeps (grown on demand, bounded per call).
#include <algorithm>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/swb200.h"
#include "sw_device.cuh"
#include "sw_engine.h"

using namespace swb;

namespace {

constexpr int kTbRows = 4;                     // query rows per lane
constexpr int kTbWarpRows = 32 * kTbRows;      // rows per warp
constexpr int kTbMaxWarps = 32;                // warps (row blocks in flight) per record
constexpr int kTbK = 32;                       // column steps between block barriers
// Step lag of warp w behind warp w-1: its last lane writes column c at its
// step c + 31, the next warp's first lane reads it a step ahead of its own, at
// c - 1, which is K block steps later, so a barrier lies between; the entry's next
// write (column c + 128) comes 96 >= K steps after that read, past another.
constexpr int kTbLag = kTbK + 32;
constexpr int kTbRing = 128;
constexpr int kTbLimitRows = 512;              // row granularity of the size limit
constexpr int kTbNeg = -(1 << 28);             // below any reachable E/F
constexpr size_t kTbMaxScratch = (size_t)8 << 30;   // direction bits + boundary rows per call

struct TbJob {
    uint32_t pos;          // sorted position of the record (pair = pos / 2, half = pos % 2)
    uint32_t dlen;         // record length
    uint64_t dir;          // first direction word
    uint64_t bnd;          // first boundary entry (int2 units)
    uint64_t ops;          // first op byte
};

struct TbOut {
    int32_t score;
    uint32_t q_begin, q_end, d_begin, d_end;
    uint32_t n_ops, matches, pad;
};

struct TbArgs {
    const uint8_t* db;     // the resident column streams, as bytes
    const Pair2* pairs;
    const uint8_t* query;
    int qlen;
    const int8_t* mat;
    int gap_oe, gap_e;
    int n;
    const TbJob* jobs;
    uint16_t* dir;
    int2* bnd;
    uint8_t* ops;          // per job: qlen + dlen bytes, written last op first
    TbOut* out;
};

// Steps of a warp over a record: its columns and the lanes' skew, in whole
// barrier intervals.
__host__ __device__ constexpr int tb_span(int dlen) {
    return (dlen + 31 + kTbK - 1) / kTbK * kTbK;
}

// The direction bits of a cell: bit 3 - k of a word's four nibbles for row k of
// a lane's 4 (four words of their own while a column is scored: one would be a
// chain of 16 shifts).
constexpr uint32_t kTbNotDiag = 1u, kTbNotE = 1u << 4, kTbExtE = 1u << 8, kTbExtF = 1u << 12;

// Row i, column j's bits (at the masks above).  A warp's lanes store their words side by side, step
// by step (step = column + lane).
__device__ __forceinline__ uint32_t tb_bits(const uint16_t* dir, int span, int i, int j) {
    const int row_block = i / kTbRows, lane = row_block & 31;
    const uint32_t w = dir[((size_t)(row_block >> 5) * span + j + lane) * 32 + lane];
    return w >> (kTbRows - 1 - i % kTbRows);
}

struct TbBest {
    int score, col, row;
};

__device__ __forceinline__ void tb_better(TbBest& b, int score, int col, int row) {
    if (score > b.score ||
        (score == b.score && (col < b.col || (col == b.col && row < b.row))))
        b = TbBest{score, col, row};
}

// bits << 1 | (x < 0)
__device__ __forceinline__ uint32_t tb_sign_in(uint32_t bits, int x) {
    return __funnelshift_l((uint32_t)x, bits, 1);
}

// Dynamic shared memory: per warp a profile of its rows (4 signed bytes per
// code and lane) and the ring it writes.
constexpr size_t kTbProfWords = 25 * 32;
constexpr size_t tb_smem(int warps) {
    return warps * (kTbProfWords * sizeof(uint32_t) + kTbRing * sizeof(int2));
}

__global__ void __launch_bounds__(32 * kTbMaxWarps) sw_traceback_kernel(const TbArgs a) {
    extern __shared__ uint32_t tb_shared[];
    __shared__ TbBest s_best[kTbMaxWarps];
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
    const int warps = (int)(blockDim.x >> 5);
    const TbJob job = a.jobs[blockIdx.x];
    const int dlen = (int)job.dlen;
    const int qlen = a.qlen;
    const uint8_t* rec = a.db + (size_t)a.pairs[job.pos >> 1].off16 * 16 + (job.pos & 1);
    uint16_t* dir = a.dir + job.dir;
    int2* bnd = a.bnd + job.bnd;
    uint32_t* const prof = tb_shared + w * kTbProfWords;
    int2* const rings = reinterpret_cast<int2*>(tb_shared + warps * kTbProfWords);
    int2* const ring_out = rings + w * kTbRing;
    const int2* const ring_in = rings + (w > 0 ? w - 1 : 0) * kTbRing;
    const int blocks = (qlen + kTbWarpRows - 1) / kTbWarpRows;      // 128-row blocks
    const int span = tb_span(dlen);
    TbBest best{0, 0x7fffffff, 0x7fffffff};
    for (int base = 0; base < blocks; base += warps) {
        const int rb = base + w;                                    // this warp's block
        const bool active = rb < blocks;
        const bool from_bnd = w == 0 && base > 0;
        const bool to_bnd = w == warps - 1 && rb + 1 < blocks;
        const int r0 = rb * kTbWarpRows + lane * kTbRows;
        __syncthreads();                 // the previous row blocks are done
        if (active)
            for (int i = 0; i < 25; ++i) {
                uint32_t v = 0;
#pragma unroll
                for (int k = 0; k < kTbRows; ++k)
                    if (r0 + k < qlen)
                        v |= (uint32_t)(uint8_t)a.mat[(a.query[r0 + k] & 31) * 32 + i] << (8 * k);
                prof[i * 32 + lane] = v;
            }
        __syncthreads();
        int H[kTbRows], E[kTbRows];
#pragma unroll
        for (int k = 0; k < kTbRows; ++k) {
            H[k] = 0;
            E[k] = kTbNeg;
        }
        int out_h = 0, out_f = kTbNeg, prev_h = 0;
        const int used = min(warps, blocks - base);
        const int total = (used - 1) * kTbLag + span;
        uint16_t* dw = dir + (size_t)rb * span * 32 + lane;
        // Rows past the query score 0 and never come first: their H is at most
        // an earlier column's.
        TbBest mine{0, 0x7fffffff, 0x7fffffff};    // of this lane's rows: columns ascend
        auto residue = [&](int c) { return c >= 0 && c < dlen ? (unsigned)rec[2 * (size_t)c] : 24u; };
        unsigned code = residue(1 - lane);
        uint32_t p = prof[min(residue(-lane), 24u) * 32 + lane];
        int2 up = make_int2(0, kTbNeg);            // lane 0: the row above, this step's column
        for (int gs = 0; gs < total; gs += kTbK) {
            const int s0 = gs - w * kTbLag;        // this warp's first step of the interval
            if (active && s0 >= 0 && s0 < span) {  // warp-uniform; whole intervals
                if (s0 == 0 && w > 0) up = ring_in[0];
                if (s0 == 0 && from_bnd && dlen > 0) up = bnd[0];
                for (int s = s0; s < s0 + kTbK; ++s) {
                    const int c = s - lane;
                    int h_in = __shfl_up_sync(FULL, out_h, 1);
                    int f_in = __shfl_up_sync(FULL, out_f, 1);
                    const bool above = lane == 0 && c < dlen;
                    h_in = above ? up.x : lane == 0 ? 0 : h_in;
                    f_in = above ? up.y : lane == 0 ? kTbNeg : f_in;
                    // the next step's row above (written K or more block steps
                    // ago), profile word and residue
                    if (w > 0) up = ring_in[(s + 1) & (kTbRing - 1)];
                    if (from_bnd && s + 1 < dlen) up = bnd[s + 1];
                    const uint32_t p_next = prof[min(code, 24u) * 32 + lane];
                    code = residue(c + 2);
                    int hd[kTbRows];
#pragma unroll
                    for (int k = 0; k < kTbRows; ++k)
                        hd[k] = (k > 0 ? H[k > 0 ? k - 1 : 0] : prev_h) +
                                (int)(int8_t)(p >> (8 * k));
                    int f = f_in;
                    uint32_t b_diag = 0u, b_e = 0u, b_ee = 0u, b_ef = 0u;
#pragma unroll
                    for (int k = 0; k < kTbRows; ++k) {
                        const int t = __vimax3_s32(hd[k], E[k], 0);
                        const int h = max(t, f);
                        const int o = h - a.gap_oe, ee = E[k] - a.gap_e, fe = f - a.gap_e;
                        b_diag = tb_sign_in(b_diag, hd[k] - h);
                        b_e = tb_sign_in(b_e, E[k] - h);
                        b_ee = tb_sign_in(b_ee, o - ee);
                        b_ef = tb_sign_in(b_ef, o - fe);
                        E[k] = max(o, ee);
                        f = max(t - a.gap_oe, fe);
                        H[k] = h;
                    }
                    static_assert(kTbRows == 4, "the maximum below, the bits' and profile's words");
                    const int m = __vimax3_s32(max(H[0], H[1]), H[2], H[3]);
                    if (m > mine.score) {
                        int row = kTbRows - 1;
#pragma unroll
                        for (int k = kTbRows - 2; k >= 0; --k) row = H[k] == m ? k : row;
                        mine = TbBest{m, c, r0 + row};
                    }
                    out_h = H[kTbRows - 1];
                    out_f = f;
                    *dw = (uint16_t)(b_diag | b_e << 4 | b_ee << 8 | b_ef << 12);
                    dw += 32;
                    if (lane == 31 && c >= 0) {
                        if (w + 1 < warps) ring_out[c & (kTbRing - 1)] = make_int2(out_h, out_f);
                        if (to_bnd && c < dlen) bnd[c] = make_int2(out_h, out_f);
                    }
                    prev_h = h_in;
                    p = p_next;
                }
            }
            __syncthreads();
        }
        tb_better(best, mine.score, mine.col, mine.row);
    }
    // end cell: maximal score, then smallest record position, then smallest row
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        tb_better(best, __shfl_xor_sync(FULL, best.score, o), __shfl_xor_sync(FULL, best.col, o),
                  __shfl_xor_sync(FULL, best.row, o));
    if (lane == 0) s_best[w] = best;
    __syncthreads();         // and every direction word is visible to warp 0
    if (w != 0) return;
    for (int i = 0; i < warps; ++i) tb_better(best, s_best[i].score, s_best[i].col, s_best[i].row);
    TbOut o{};
    o.score = best.score;
    if (best.score > 0) {
        uint8_t* ops = a.ops + job.ops;
        int i = best.row, j = best.col, si = i, sj = j, hv = best.score;   // hv: H at (i, j)
        uint32_t n = 0, matches = 0;
        while (true) {
            // the diagonal from (i, j): lane l looks at (i - l, j - l), whose H
            // is hv less the scores of the lanes before it
            const int ii = i - lane, jj = j - lane;
            const bool valid = ii >= 0 && jj >= 0;
            const int qr = valid ? a.query[ii] & 31 : 0, dr = valid ? rec[2 * (size_t)jj] & 31 : 0;
            const int p = valid ? a.mat[qr * 32 + dr] : 0;
            const uint32_t bits = valid ? tb_bits(dir, span, ii, jj) : kTbNotDiag;
            int sum = p;
#pragma unroll
            for (int x = 1; x < 32; x <<= 1) {
                const int y = __shfl_up_sync(FULL, sum, x);
                if (lane >= x) sum += y;
            }
            const unsigned stop =
                ~__ballot_sync(FULL, valid && !(bits & kTbNotDiag) && hv - (sum - p) > 0);
            const int run = stop ? __ffs(stop) - 1 : 32;
            matches += __popc(__ballot_sync(FULL, qr == dr && lane < run));
            if (lane < run) ops[n + lane] = 0;
            if (run > 0) {
                hv -= __shfl_sync(FULL, sum, run - 1);
                si = i - (run - 1);
                sj = j - (run - 1);
                i -= run;
                j -= run;
                n += run;
            }
            if (run == 32) continue;
            if (hv <= 0 || i < 0 || j < 0) break;
            const bool e_gap = !(__shfl_sync(FULL, bits, run) & kTbNotE);
            while (true) {                   // the gap's cells, up to the one that opened it
                const int ci = e_gap ? i : i - 1 - lane, cj = e_gap ? j - 1 - lane : j;
                const bool opened = ci < 0 || cj < 0 ||
                                    !(tb_bits(dir, span, ci, cj) & (e_gap ? kTbExtE : kTbExtF));
                const unsigned open = __ballot_sync(FULL, opened);
                const int len = open ? __ffs(open) : 32;
                if (lane < len) ops[n + lane] = e_gap ? 2 : 1;
                n += len;
                hv += len * a.gap_e;
                if (e_gap) j -= len;
                else i -= len;
                if (open) break;
            }
            hv += a.gap_oe - a.gap_e;
        }
        o.q_begin = (uint32_t)si;
        o.q_end = (uint32_t)best.row + 1;
        o.d_begin = (uint32_t)sj;
        o.d_end = (uint32_t)best.col + 1;
        o.n_ops = n;
        o.matches = matches;
    }
    if (lane == 0) a.out[blockIdx.x] = o;
}

template <typename T>
cudaError_t grow(T** p, size_t& cap, size_t need) {
    if (need <= cap) return cudaSuccess;
    dev_free(*p);
    cap = 0;
    cudaError_t e = dev_alloc(p, need);
    if (e == cudaSuccess) cap = need;
    return e;
}

}  // namespace

struct sw_tb_state {
    uint16_t* d_dir = nullptr;
    size_t dir_cap = 0;
    int2* d_bnd = nullptr;
    size_t bnd_cap = 0;
    uint8_t* d_ops = nullptr;
    size_t ops_cap = 0;
    TbJob* d_jobs = nullptr;
    size_t jobs_cap = 0;
    TbOut* d_out = nullptr;
    size_t out_cap = 0;
};

namespace swb {
void free_traceback(sw_ctx* ctx) {
    sw_tb_state* t = ctx->tb;
    if (!t) return;
    dev_free(t->d_dir);
    dev_free(t->d_bnd);
    dev_free(t->d_ops);
    dev_free(t->d_jobs);
    dev_free(t->d_out);
    delete t;
    ctx->tb = nullptr;
}
}  // namespace swb

extern "C" sw_status sw_traceback(sw_ctx* ctx, const uint8_t* query, uint32_t qlen,
                                  const uint64_t* records, uint32_t n, sw_alignment* out,
                                  uint32_t* ops, uint64_t ops_cap, uint64_t* ops_used) {
    if (!ctx) return SW_ERR_INVALID;
    if (ctx->serve) return SW_ERR_BUSY;   // the serving loop owns the stream
    if (!ctx->db_loaded) SW_SET(ctx, SW_ERR_STATE, "no DB loaded (call sw_db_load first)");
    if (!ops_used || (n && (!records || !out)) || (qlen && !query))
        SW_SET(ctx, SW_ERR_INVALID, "null argument");
    *ops_used = 0;
    if (n == 0) return SW_OK;
    for (uint32_t i = 0; i < qlen; ++i)
        if (query[i] > 24) SW_SET(ctx, SW_ERR_INVALID, "query code %d at %u", query[i], i);
    for (uint32_t h = 0; h < n; ++h) {
        if (records[h] >= (uint64_t)ctx->n_records)
            SW_SET(ctx, SW_ERR_INVALID, "record %llu out of range",
                   (unsigned long long)records[h]);
        out[h] = sw_alignment{};
        out[h].index = records[h];
    }
    if (qlen == 0) return SW_OK;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    if (!ctx->tb) ctx->tb = new sw_tb_state();
    sw_tb_state* tb = ctx->tb;
    const uint64_t blocks = (qlen + kTbWarpRows - 1) / kTbWarpRows;
    const int warps = (int)std::min<uint64_t>(blocks, kTbMaxWarps);
    const uint64_t P = (qlen + kTbLimitRows - 1) / kTbLimitRows;    // for the size limit
    // jobs in rounds whose scratch fits the per-call bound
    std::vector<TbJob> jobs(n);
    std::vector<TbOut> res(n);
    uint64_t ops_total = 0;
    for (uint32_t h = 0; h < n; ++h) {
        const uint64_t dlen = ctx->rec_len[records[h]];
        const size_t need = (size_t)(P * 32 * dlen) * sizeof(uint2) + dlen * sizeof(int2);
        if (need > kTbMaxScratch)
            SW_SET(ctx, SW_ERR_UNSUPPORTED,
                   "traceback of a %u x %llu matrix needs %zu bytes of direction bits (limit %zu)",
                   qlen, (unsigned long long)dlen, need, kTbMaxScratch);
        jobs[h].pos = ctx->rec_pos[records[h]];
        jobs[h].dlen = (uint32_t)dlen;
    }
    std::vector<uint8_t> hops;
    uint32_t h0 = 0;
    while (h0 < n) {
        uint64_t dir = 0, bnd = 0, opsb = 0;
        uint32_t h1 = h0;
        while (h1 < n) {
            const uint64_t dlen = jobs[h1].dlen;
            const uint64_t ndir = blocks * 32 * tb_span((int)dlen), nbnd = dlen;
            if (h1 > h0 &&
                (dir + ndir) * sizeof(uint16_t) + (bnd + nbnd) * sizeof(int2) > kTbMaxScratch)
                break;
            jobs[h1].dir = dir;
            jobs[h1].bnd = bnd;
            jobs[h1].ops = opsb;
            dir += ndir;
            bnd += nbnd;
            opsb += qlen + dlen;
            ++h1;
        }
        const uint32_t m = h1 - h0;
        cudaStream_t st = ctx->stream;
        sw_status s = ensure_query_buffers(ctx, qlen);
        if (s != SW_OK) return s;
        memcpy(ctx->h_query, query, qlen);
        if (grow(&tb->d_dir, tb->dir_cap, std::max<uint64_t>(dir, 1)) != cudaSuccess ||
            grow(&tb->d_bnd, tb->bnd_cap, std::max<uint64_t>(bnd, 1)) != cudaSuccess ||
            grow(&tb->d_ops, tb->ops_cap, std::max<uint64_t>(opsb, 1)) != cudaSuccess ||
            grow(&tb->d_jobs, tb->jobs_cap, m) != cudaSuccess ||
            grow(&tb->d_out, tb->out_cap, m) != cudaSuccess)
            SW_SET(ctx, SW_ERR_NOMEM, "device allocation failed: traceback scratch");
        SW_CUDA(ctx, cudaMemcpyAsync(ctx->d_query, ctx->h_query, qlen, cudaMemcpyHostToDevice, st));
        SW_CUDA(ctx, cudaMemcpyAsync(tb->d_jobs, jobs.data() + h0, m * sizeof(TbJob),
                                     cudaMemcpyHostToDevice, st));
        TbArgs a;
        a.db = reinterpret_cast<const uint8_t*>(ctx->d_db);
        a.pairs = ctx->d_pairs;
        a.query = ctx->d_query;
        a.qlen = (int)qlen;
        a.mat = ctx->d_mat;
        a.gap_oe = ctx->params.gap_open + ctx->params.gap_extend;
        a.gap_e = ctx->params.gap_extend;
        a.n = (int)m;
        a.jobs = tb->d_jobs;
        a.dir = tb->d_dir;
        a.bnd = tb->d_bnd;
        a.ops = tb->d_ops;
        a.out = tb->d_out;
        void* args[] = {&a};
        SW_CUDA(ctx, cudaFuncSetAttribute((const void*)sw_traceback_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)tb_smem(kTbMaxWarps)));
        SW_CUDA(ctx, cudaLaunchKernel((const void*)sw_traceback_kernel, dim3(m), dim3(32 * warps),
                                      args, tb_smem(warps), st));
        SW_CUDA(ctx, cudaMemcpyAsync(res.data() + h0, tb->d_out, m * sizeof(TbOut),
                                     cudaMemcpyDeviceToHost, st));
        hops.resize(opsb);
        SW_CUDA(ctx, cudaMemcpyAsync(hops.data(), tb->d_ops, opsb, cudaMemcpyDeviceToHost, st));
        SW_CUDA(ctx, cudaStreamSynchronize(st));
        SW_CUDA(ctx, cudaGetLastError());
        // ops were written last first: run-length encode them in alignment order
        for (uint32_t h = h0; h < h1; ++h) {
            const TbOut& r = res[h];
            sw_alignment& al = out[h];
            al.score = r.score;
            al.q_begin = r.q_begin;
            al.q_end = r.q_end;
            al.d_begin = r.d_begin;
            al.d_end = r.d_end;
            al.matches = r.matches;
            al.ops_offset = ops_total;
            const uint8_t* o = hops.data() + jobs[h].ops;
            uint32_t runs = 0;
            for (int64_t x = (int64_t)r.n_ops - 1; x >= 0;) {
                const uint8_t op = o[x];
                uint32_t len = 0;
                while (x >= 0 && o[x] == op) {
                    ++len;
                    --x;
                }
                if (ops && ops_total < ops_cap) ops[ops_total] = (len << 4) | op;
                ++ops_total;
                ++runs;
            }
            al.n_ops = runs;
        }
        h0 = h1;
    }
    *ops_used = ops_total;
    if (ops_total > ops_cap)
        SW_SET(ctx, SW_ERR_UNSUPPORTED, "ops buffer too small: %llu entries needed",
               (unsigned long long)ops_total);
    return SW_OK;
}
