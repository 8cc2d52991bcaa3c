// sw_engine.cu -- host side of libswb200: context, resident DB layout, kernel
// shape selection and the plain search sequence behind the C ABI (swb200.h).
//
// Reference flow this replaces (SWhybrid, CUDA build): per query and per
// 256 MB chunk, DataPool::fillChunk reads batches from disk, CUDAWorker::packDB
// re-packs them on the host, asyncCopy ships the whole chunk over PCIe,
// kernelLaunch runs, and a synchronous cudaMemcpy brings the scores back
// (src/Worker.cpp:175-200, src/CUDAWorker.cu:144-246); overflowed records are
// re-scored on the host afterwards (src/RecalcWorker.cpp:99-268) and top-k is
// merged by list insertion (src/ResultList.h:37-79).
//
// Here the DB is laid out once (sorted by length, paired, column-interleaved)
// and stays in HBM; a search is: query H2D (a few KB), first-pass kernel(s),
// 32-bit re-score of the flagged records, device top-k, D2H of k hits.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <iterator>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/swb200.h"
#include "sw_aux.h"
#include "sw_device.cuh"
#include "sw_engine.h"
#include "sw_long.h"
#include "sw_tuned_default.h"
#include "sw_registry.h"

namespace swb {
int plain_cell(int lo, int hi, int q, int e);
extern const WfKernel wf_table_t4[];
extern const int wf_table_t4_n;
extern const WfKernel wf_table_t8[];
extern const int wf_table_t8_n;
extern const WfKernel wf_table_t16[];
extern const int wf_table_t16_n;
extern const WfKernel wf_table_t32[];
extern const int wf_table_t32_n;

const WfKernel* wf_kernels(int* n) {
    static std::vector<WfKernel> all;
    static std::once_flag once;
    std::call_once(once, [] {
        auto add = [](const WfKernel* t, int m) { all.insert(all.end(), t, t + m); };
        add(wf_table_t4, wf_table_t4_n);
        add(wf_table_t8, wf_table_t8_n);
        add(wf_table_t16, wf_table_t16_n);
        add(wf_table_t32, wf_table_t32_n);
    });
    *n = (int)all.size();
    return all.data();
}

const WfKernel* find_kernel(int T, int R) {
    int n = 0;
    const WfKernel* k = wf_kernels(&n);
    for (int i = 0; i < n; ++i)
        if (k[i].T == T && k[i].R == R) return &k[i];
    return nullptr;
}

}  // namespace swb

using namespace swb;

namespace {

constexpr int kMinWindow = 256;     // shortest window of a long pair, in columns

double now_ms() {
    return std::chrono::duration<double, std::milli>(
               std::chrono::steady_clock::now().time_since_epoch())
        .count();
}

}  // namespace

// ---------------------------------------------------------------------------
// parameters and encoding
// ---------------------------------------------------------------------------

// BLOSUM62 in the reference's code order (A B C D E F G H I K L M N P Q R S T
// V W X Y Z), the table of src/Param.h:8-51.  Rows/columns 23..31 are zero.
static const int8_t kBlosum62[23][23] = {
    {4, -2, 0, -2, -1, -2, 0, -2, -1, -1, -1, -1, -2, -1, -1, -1, 1, 0, 0, -3, 0, -2, -1},
    {-2, 4, -3, 4, 1, -3, -1, 0, -3, 0, -4, -3, 3, -2, 0, -1, 0, -1, -3, -4, -1, -3, 1},
    {0, -3, 9, -3, -4, -2, -3, -3, -1, -3, -1, -1, -3, -3, -3, -3, -1, -1, -1, -2, -2, -2, -3},
    {-2, 4, -3, 6, 2, -3, -1, -1, -3, -1, -4, -3, 1, -1, 0, -2, 0, -1, -3, -4, -1, -3, 1},
    {-1, 1, -4, 2, 5, -3, -2, 0, -3, 1, -3, -2, 0, -1, 2, 0, 0, -1, -2, -3, -1, -2, 4},
    {-2, -3, -2, -3, -3, 6, -3, -1, 0, -3, 0, 0, -3, -4, -3, -3, -2, -2, -1, 1, -1, 3, -3},
    {0, -1, -3, -1, -2, -3, 6, -2, -4, -2, -4, -3, 0, -2, -2, -2, 0, -2, -3, -2, -1, -3, -2},
    {-2, 0, -3, -1, 0, -1, -2, 8, -3, -1, -3, -2, 1, -2, 0, 0, -1, -2, -3, -2, -1, 2, 0},
    {-1, -3, -1, -3, -3, 0, -4, -3, 4, -3, 2, 1, -3, -3, -3, -3, -2, -1, 3, -3, -1, -1, -3},
    {-1, 0, -3, -1, 1, -3, -2, -1, -3, 5, -2, -1, 0, -1, 1, 2, 0, -1, -2, -3, -1, -2, 1},
    {-1, -4, -1, -4, -3, 0, -4, -3, 2, -2, 4, 2, -3, -3, -2, -2, -2, -1, 1, -2, -1, -1, -3},
    {-1, -3, -1, -3, -2, 0, -3, -2, 1, -1, 2, 5, -2, -2, 0, -1, -1, -1, 1, -1, -1, -1, -1},
    {-2, 3, -3, 1, 0, -3, 0, 1, -3, 0, -3, -2, 6, -2, 0, 0, 1, 0, -3, -4, -1, -2, 0},
    {-1, -2, -3, -1, -1, -4, -2, -2, -3, -1, -3, -2, -2, 7, -1, -2, -1, -1, -2, -4, -2, -3, -1},
    {-1, 0, -3, 0, 2, -3, -2, 0, -3, 1, -2, 0, 0, -1, 5, 1, 0, -1, -2, -2, -1, -1, 3},
    {-1, -1, -3, -2, 0, -3, -2, 0, -3, 2, -2, -1, 0, -2, 1, 5, -1, -1, -3, -3, -1, -2, 0},
    {1, 0, -1, 0, 0, -2, 0, -1, -2, 0, -2, -1, 1, -1, 0, -1, 4, 1, -2, -3, 0, -2, 0},
    {0, -1, -1, -1, -1, -2, -2, -2, -1, -1, -1, -1, 0, -1, -1, -1, 1, 5, 0, -2, 0, -2, -1},
    {0, -3, -1, -3, -2, -1, -3, -3, 3, -2, 1, 1, -3, -2, -2, -3, -2, 0, 4, -3, -1, -1, -2},
    {-3, -4, -2, -4, -3, 1, -2, -2, -3, -3, -2, -1, -4, -4, -2, -3, -3, -2, -3, 11, -2, 2, -3},
    {0, -1, -2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -2, -1, -1, 0, 0, -1, -2, -1, -1, -1},
    {-2, -3, -2, -3, -2, 3, -3, 2, -1, -2, -1, -1, -2, -3, -1, -2, -2, -2, -1, 2, -1, 7, -2},
    {-1, 1, -3, 1, 4, -3, -2, 0, -3, 1, -3, -1, 0, -1, 3, 0, 0, -1, -2, -3, -1, -2, 4},
};

extern "C" void sw_params_default(sw_params* p) {
    if (!p) return;
    memset(p, 0, sizeof(*p));
    for (int i = 0; i < 23; ++i)
        for (int j = 0; j < 23; ++j) p->matrix[i * 32 + j] = kBlosum62[i][j];
    p->gap_open = 10;
    p->gap_extend = 2;
    p->top_k = 10;
    p->flags = SW_FLAG_REFERENCE_CAP;
}

extern "C" sw_status sw_encode(const char* letters, uint64_t n, uint8_t* codes) {
    if ((!letters || !codes) && n) return SW_ERR_INVALID;
    static const char* alpha = "ABCDEFGHIKLMNPQRSTVWXYZ";
    uint8_t tab[256];
    memset(tab, kZeroCode, sizeof(tab));
    for (int i = 0; alpha[i]; ++i) {
        tab[(uint8_t)alpha[i]] = (uint8_t)i;
        tab[(uint8_t)(alpha[i] - 'A' + 'a')] = (uint8_t)i;
    }
    tab[(uint8_t)'@'] = 23;
    for (uint64_t i = 0; i < n; ++i) codes[i] = tab[(uint8_t)letters[i]];
    return SW_OK;
}

// ---------------------------------------------------------------------------
// context
// ---------------------------------------------------------------------------

extern "C" const char* sw_last_error(const sw_ctx* ctx) {
    return ctx ? ctx->err.c_str() : swb::thread_error();
}

static sw_status validate_params(sw_ctx* ctx, const sw_params* p) {
    if (p->gap_open < 0 || p->gap_extend < 0 || p->gap_open + p->gap_extend > 1000)
        SW_SET(ctx, SW_ERR_INVALID, "gap costs out of range (open %d, extend %d)", p->gap_open,
               p->gap_extend);
    if (p->top_k < 1 || p->top_k > kMaxTopK)
        SW_SET(ctx, SW_ERR_INVALID, "top_k %d outside 1..%d", p->top_k, kMaxTopK);
    for (int i = 0; i < 1024; ++i)
        if (p->matrix[i] < -127 || p->matrix[i] > 127)
            SW_SET(ctx, SW_ERR_INVALID, "matrix entry %d = %d outside -127..127", i,
                   p->matrix[i]);
    return SW_OK;
}

extern "C" sw_status sw_ctx_create(int device, const sw_params* params, sw_ctx** out) {
    if (!out) return SW_ERR_INVALID;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return SW_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= ndev) return SW_ERR_INVALID;
    sw_ctx* ctx = new sw_ctx();
    ctx->device = device;
    if (params) ctx->params = *params;
    else sw_params_default(&ctx->params);
    sw_status st = validate_params(ctx, &ctx->params);
    if (st != SW_OK) {
        delete ctx;
        return st;
    }
    auto fail = [&](sw_status s) {
        cudaGetLastError();     // a refused call must not surface in the caller's next one
        sw_ctx_destroy(ctx);
        return s;
    };
    if (cudaSetDevice(device) != cudaSuccess) return fail(SW_ERR_CUDA);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return fail(SW_ERR_CUDA);
    ctx->num_sms = prop.multiProcessorCount;
    ctx->max_smem = (int)prop.sharedMemPerBlockOptin;
    ctx->regs_per_sm = prop.regsPerMultiprocessor;
    if (cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking) != cudaSuccess)
        return fail(SW_ERR_CUDA);
    ctx->stream = ctx->own_stream;
    ctx->tuning.assign(std::begin(kDefaultTuning), std::end(kDefaultTuning));
    if (cudaStreamCreateWithFlags(&ctx->side_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->fork_ev, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->join_ev, cudaEventDisableTiming) != cudaSuccess)
        return fail(SW_ERR_CUDA);
    for (auto& e : ctx->ev)
        if (cudaEventCreate(&e) != cudaSuccess) return fail(SW_ERR_CUDA);
    // matrix: int8 copy; codes >= 24 (zero code, pads) score 0
    int8_t mat8[1024];
    int lo = 0, hi = 0;
    for (int i = 0; i < 32; ++i)
        for (int j = 0; j < 32; ++j) {
            int v = (i >= kZeroCode || j >= kZeroCode) ? 0 : ctx->params.matrix[i * 32 + j];
            mat8[i * 32 + j] = (int8_t)v;
            lo = std::min(lo, v);
            hi = std::max(hi, v);
            ctx->row_best[i] = std::max(ctx->row_best[i], v);
        }
    ctx->max_score = hi;
    ctx->cell = plain_cell(lo, hi, ctx->params.gap_open + ctx->params.gap_extend,
                           ctx->params.gap_extend);
    if (dev_alloc(&ctx->d_mat, 1024) != cudaSuccess) return fail(SW_ERR_NOMEM);
    if (cudaMemcpy(ctx->d_mat, mat8, 1024, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(SW_ERR_CUDA);
    // every first-pass kernel may use the opt-in shared-memory maximum, less
    // what it holds statically (the long-pair kernels hold a few words)
    auto allow_smem = [&](const void* fn) {
        cudaFuncAttributes fa;
        return cudaFuncGetAttributes(&fa, fn) == cudaSuccess &&
               cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    ctx->max_smem - (int)fa.sharedSizeBytes) == cudaSuccess;
    };
    // what the kernels' registers and static shared memory allow, for the layout
    // of each search
    int nk = 0;
    const WfKernel* ks = wf_kernels(&nk);
    for (int i = 0; i < nk; ++i) {
        sw_ctx::PlainFit f;
        const void* fns[2] = {ks[i].fn[ctx->cell], ks[i].batch_fn};
        const int blocks[2] = {plain_block(ctx, ks[i]), ks[i].block};
        for (int v = 0; v < 2; ++v) {
            cudaFuncAttributes fa;
            if (!allow_smem(fns[v]) || cudaFuncGetAttributes(&fa, fns[v]) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f.blocks[v], fns[v], blocks[v], 0) !=
                    cudaSuccess)
                return fail(SW_ERR_CUDA);
            f.max_dyn[v] = ctx->max_smem - (int)fa.sharedSizeBytes;
        }
        ctx->plain_fit.push_back(f);
    }
    const QpKernel* qks = qp_kernels(&nk);
    for (int i = 0; i < nk; ++i)
        if (!allow_smem(qks[i].fn[ctx->cell])) return fail(SW_ERR_CUDA);
    const LongKernel* lks = long_kernels(&nk);
    for (int i = 0; i < nk; ++i) {
        cudaFuncAttributes fa;
        if (!allow_smem(lks[i].fn[ctx->cell]) ||
            cudaFuncGetAttributes(&fa, lks[i].fn[ctx->cell]) != cudaSuccess)
            return fail(SW_ERR_CUDA);
        ctx->long_fit.push_back({fa.numRegs, ctx->max_smem - (int)fa.sharedSizeBytes});
    }
    if (!allow_smem(long_item_kernel().fn[ctx->cell])) return fail(SW_ERR_CUDA);
    *out = ctx;
    return SW_OK;
}

static void free_db_buffers(sw_ctx* ctx) {
    dev_free(ctx->d_rs_scratch);
    dev_free(ctx->d_db);
    dev_free(ctx->d_pairs);
    dev_free(ctx->d_win_pairs);
    dev_free(ctx->d_win_ids);
    dev_free(ctx->d_perm);
    dev_free(ctx->d_bnd);
    dev_free(ctx->d_counters);
    ctx->d_scores = nullptr;
    dev_free(ctx->d_scores_rec);
    dev_free(ctx->d_ovf);
    dev_free(ctx->d_keys[0]);
    dev_free(ctx->d_keys[1]);
}

static void free_db(sw_ctx* ctx) {
    swb::free_batch(ctx);
    swb::free_traceback(ctx);
    swb::free_image(ctx);
    ctx->rec_pos.clear();
    ctx->rec_len.clear();
    free_db_buffers(ctx);
    ctx->n_records = 0;
    ctx->n_pairs = 0;
    ctx->pair_ncols.clear();
    ctx->pair_prefix.clear();
    ctx->db_loaded = false;
}

extern "C" sw_status sw_ctx_destroy(sw_ctx* ctx) {
    if (!ctx) return SW_ERR_INVALID;
    cudaSetDevice(ctx->device);
    serve_teardown(ctx);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->own_stream) cudaStreamSynchronize(ctx->own_stream);
    if (ctx->side_stream) cudaStreamSynchronize(ctx->side_stream);
    free_db(ctx);
    dev_free(ctx->d_mat);
    dev_free(ctx->d_query);
    if (ctx->h_query) cudaFreeHost(ctx->h_query);
    if (ctx->h_keys) cudaFreeHost(ctx->h_keys);
    for (auto& e : ctx->ev)
        if (e) cudaEventDestroy(e);
    for (auto* v : {&ctx->pending, &ctx->spare})
        for (auto& m : *v)
            for (auto& e : m.e) cudaEventDestroy(e);
    if (ctx->fork_ev) cudaEventDestroy(ctx->fork_ev);
    if (ctx->join_ev) cudaEventDestroy(ctx->join_ev);
    if (ctx->side_stream) cudaStreamDestroy(ctx->side_stream);
    if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
    delete ctx;
    return SW_OK;
}

// ---------------------------------------------------------------------------
// database layout
// ---------------------------------------------------------------------------

extern "C" sw_status sw_db_load(sw_ctx* ctx, const uint8_t* residues, const uint64_t* offsets,
                                uint64_t n) {
    return swb::db_load(ctx, residues, offsets, n, nullptr);
}

// The layout build behind sw_db_load and sw_db_load_image.  `given_order`
// (optional) is the length order stored in a DB image: used after checking
// that it is the stable longest-first permutation.
sw_status swb::db_load(sw_ctx* ctx, const uint8_t* residues, const uint64_t* offsets, uint64_t n,
                       const uint32_t* given_order) {
    if (!ctx) return SW_ERR_INVALID;
    if (ctx->serve) return SW_ERR_BUSY;   // the serving loop owns the stream and the DB
    if (!offsets || (n && !residues && offsets[n] != offsets[0]))
        SW_SET(ctx, SW_ERR_INVALID, "null residues/offsets");
    if (n >= (1ull << 31)) SW_SET(ctx, SW_ERR_UNSUPPORTED, "too many records (%llu)",
                                  (unsigned long long)n);
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    SW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    free_db(ctx);
    std::vector<uint32_t> len(n);
    uint64_t total = 0, maxlen = 0;
    for (uint64_t i = 0; i < n; ++i) {
        if (offsets[i + 1] < offsets[i]) SW_SET(ctx, SW_ERR_INVALID, "offsets not monotone at %llu",
                                                (unsigned long long)i);
        const uint64_t l = offsets[i + 1] - offsets[i];
        if (l >= (1ull << 30)) SW_SET(ctx, SW_ERR_UNSUPPORTED, "record %llu too long",
                                      (unsigned long long)i);
        len[i] = (uint32_t)l;
        total += l;
        maxlen = std::max<uint64_t>(maxlen, l);
    }
    const uint8_t* base = residues ? residues + offsets[0] : nullptr;
    for (uint64_t i = 0; i < total; ++i)
        if (base[i] > 24) SW_SET(ctx, SW_ERR_INVALID, "residue code %d at %llu (codes are 0..24)",
                                 base[i], (unsigned long long)i);
    // sort by length (longest first), stable in record order
    std::vector<uint32_t> order(n);
    if (given_order) {
        std::vector<bool> seen(n, false);
        for (uint64_t k = 0; k < n; ++k) {
            const uint32_t r = given_order[k];
            bool ok = r < n && !seen[r];
            if (ok && k > 0) {
                const uint32_t p = given_order[k - 1];
                ok = len[p] > len[r] || (len[p] == len[r] && p < r);
            }
            if (!ok) SW_SET(ctx, SW_ERR_FORMAT, "stored length order is not the stable "
                                               "longest-first permutation (entry %llu)",
                            (unsigned long long)k);
            seen[r] = true;
            order[k] = r;
        }
    } else {
        std::iota(order.begin(), order.end(), 0u);
        std::stable_sort(order.begin(), order.end(),
                         [&](uint32_t a, uint32_t b) { return len[a] > len[b]; });
    }
    const uint64_t npairs_all = (n + 1) / 2;
    std::vector<Pair2> pairs(npairs_all);
    uint64_t units = 0, nonempty = 0;
    for (uint64_t p = 0; p < npairs_all; ++p) {
        const uint32_t nc = len[order[2 * p]];
        pairs[p].off16 = (uint32_t)units;
        pairs[p].ncols = nc;
        units += (nc + 7) / 8;
        if (nc > 0) nonempty = p + 1;
        if (units >= (1ull << 32)) SW_SET(ctx, SW_ERR_UNSUPPORTED, "DB too large for 32-bit unit offsets");
    }
    int max_cols = 8;
    for (uint64_t p = 0; p < npairs_all; ++p)
        max_cols = std::max(max_cols, (int)((pairs[p].ncols + 7) / 8 * 8));
    std::vector<uint8_t> stream((size_t)units * 16, (uint8_t)kZeroCode);
    for (uint64_t p = 0; p < npairs_all; ++p) {
        uint8_t* dst = stream.data() + (size_t)pairs[p].off16 * 16;
        for (int lane = 0; lane < 2; ++lane) {
            const uint64_t k = 2 * p + lane;
            if (k >= n) break;
            const uint32_t r = order[k];
            const uint8_t* src = base + (offsets[r] - offsets[0]);
            for (uint32_t c = 0; c < len[r]; ++c) dst[2 * (size_t)c + lane] = src[c];
        }
    }
    std::vector<uint32_t> perm(n);
    for (uint64_t k = 0; k < n; ++k) perm[k] = order[k];
    ctx->rec_pos.assign(n, 0u);
    for (uint64_t k = 0; k < n; ++k) ctx->rec_pos[order[k]] = (uint32_t)k;
    ctx->rec_len = len;

    ctx->n_records = (int64_t)n;
    ctx->n_pairs = (int64_t)nonempty;
    ctx->n_residues = total;
    ctx->max_len = maxlen;
    ctx->units = units;
    ctx->pair_ncols.resize(nonempty);
    ctx->pair_prefix.assign(nonempty + 1, 0u);
    ctx->pair_cols_total = 0;
    for (uint64_t p = 0; p < nonempty; ++p) {
        ctx->pair_ncols[p] = pairs[p].ncols;
        ctx->pair_cols_total += pairs[p].ncols;
        ctx->pair_prefix[p + 1] = ctx->pair_cols_total;
    }
    ctx->db_units = (uint64_t)units;
    ctx->max_cols = max_cols;
    // room for windows of long pairs: an eighth of the DB's columns (half a
    // million for a small DB, never more than the DB itself)
    ctx->win_units = std::min<uint64_t>(units, std::max<uint64_t>(units / 8, 65536));
    // (the long-pair kernel's windows need no boundary rows, eight times as
    // much memory: twice the room)
    ctx->long_win_units = std::min<uint64_t>(units, std::max<uint64_t>(units / 4, 131072));
    // Searches do without windows where they do not fit, so a DB that nearly
    // fills the device gets no room: where it would take over half of what the
    // DB leaves free, or the buffers do not all fit beside it.
    size_t free_b = 0, total_b = 0;
    SW_CUDA(ctx, cudaMemGetInfo(&free_b, &total_b));
    const size_t nblk = (n + kTopkKeys - 1) / kTopkKeys + 1;
    const uint64_t db_need = units * 144 + npairs_all * sizeof(Pair2) + n * 16 +
                             (uint64_t)kRescoreWarps * max_cols * sizeof(uint2) +
                             2 * nblk * kMaxTopK * sizeof(unsigned long long);
    const uint64_t win_need = ctx->long_win_units * 16 + ctx->win_units * 128;
    if (units + ctx->long_win_units >= (1ull << 32) || db_need + 2 * win_need > free_b)
        ctx->win_units = ctx->long_win_units = 0;
    auto alloc = [&]() -> const char* {       // null, or what did not fit
        ctx->win_cap = (int)(ctx->long_win_units / (kMinWindow / 8) + 1);
        if (dev_alloc(&ctx->d_db, units + ctx->long_win_units) != cudaSuccess) return "db";
        if (dev_alloc(&ctx->d_win_pairs, ctx->win_cap) != cudaSuccess) return "windows";
        if (dev_alloc(&ctx->d_win_ids, ctx->win_cap) != cudaSuccess) return "windows";
        if (dev_alloc(&ctx->d_pairs, npairs_all) != cudaSuccess) return "pairs";
        if (dev_alloc(&ctx->d_perm, n) != cudaSuccess) return "perm";
        if (dev_alloc(&ctx->d_bnd, (units + ctx->win_units) * 16) != cudaSuccess)
            return "boundary rows";
        if (dev_alloc(&ctx->d_counters, kCounters + n + 1) != cudaSuccess) return "scores";
        ctx->d_scores = ctx->d_counters + kCounters;
        if (dev_alloc(&ctx->d_scores_rec, n + 1) != cudaSuccess) return "scores";
        if (dev_alloc(&ctx->d_ovf, n + 1) != cudaSuccess) return "overflow list";
        if (dev_alloc(&ctx->d_rs_scratch, (size_t)kRescoreWarps * max_cols) != cudaSuccess)
            return "re-score rows";
        if (dev_alloc(&ctx->d_keys[0], nblk * kMaxTopK) != cudaSuccess) return "keys";
        if (dev_alloc(&ctx->d_keys[1], nblk * kMaxTopK) != cudaSuccess) return "keys";
        return nullptr;
    };
    const char* failed = alloc();
    if (failed && ctx->long_win_units > 0) {
        cudaGetLastError();
        free_db_buffers(ctx);
        ctx->win_units = ctx->long_win_units = 0;
        failed = alloc();
    }
    if (failed) {
        free_db(ctx);
        cudaGetLastError();
        ctx->err = std::string("device allocation failed: ") + failed;
        return SW_ERR_NOMEM;
    }
    if (!stream.empty())
        SW_CUDA(ctx, cudaMemcpy(ctx->d_db, stream.data(), stream.size(), cudaMemcpyHostToDevice));
    if (npairs_all)
        SW_CUDA(ctx, cudaMemcpy(ctx->d_pairs, pairs.data(), npairs_all * sizeof(Pair2),
                                cudaMemcpyHostToDevice));
    if (n) SW_CUDA(ctx, cudaMemcpy(ctx->d_perm, perm.data(), n * sizeof(uint32_t),
                                   cudaMemcpyHostToDevice));
    ctx->db_bytes = (units + ctx->long_win_units) * 16 + npairs_all * sizeof(Pair2) + n * 4 +
                    (units + ctx->win_units) * 16 * 8;
    ctx->db_loaded = true;
    return SW_OK;
}

extern "C" sw_status sw_db_stats_get(const sw_ctx* ctx, sw_db_stats* out) {
    if (!ctx || !out) return SW_ERR_INVALID;
    out->n_records = (uint64_t)ctx->n_records;
    out->n_residues = ctx->n_residues;
    out->n_pairs = (uint64_t)ctx->n_pairs;
    out->max_length = ctx->max_len;
    out->device_bytes = ctx->db_bytes;
    return SW_OK;
}

// ---------------------------------------------------------------------------
// kernel shape selection
// ---------------------------------------------------------------------------

namespace swb {

// The plain kernel's cell variant for a matrix with entries lo..hi (the zero
// of unscored codes included) and gap costs q = open+extend, e = extend.
// CellNarrow's profile bytes are P + q, kept in 0..127 so that PRMT's sign
// extension leaves them unsigned; any other matrix takes CellWide.
int plain_cell(int lo, int hi, int q, int e) {
    if (lo < -q || hi > 127 - q) return kCellWide;
    if (q == 12 && e == 2) return kCellNarrow12_2;
    if (q == 12 && e == 1) return kCellNarrow12_1;
    return kCellNarrow;
}

// Blocks per SM for a kernel (v: 0 plain, 1 stacked) of a shape at a query
// length (0 = does not fit).  The runtime is asked only where shared memory
// can make a difference: it takes about a microsecond, and a layout looks at a
// dozen shapes.
static int kernel_occupancy(sw_ctx* ctx, const WfKernel& k, int v, int qlen) {
    int n = 0;
    const sw_ctx::PlainFit& f = ctx->plain_fit[&k - wf_kernels(&n)];
    const size_t smem = k.smem(qlen);
    if (smem > (size_t)f.max_dyn[v]) return 0;
    if (f.blocks[v] <= 1) return f.blocks[v];
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &nb, v ? k.batch_fn : k.fn[ctx->cell], v ? k.block : plain_block(ctx, k), smem) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return nb;
}

int shape_occupancy(sw_ctx* ctx, const WfKernel& k, int qlen) {
    return kernel_occupancy(ctx, k, 1, qlen);
}

int plain_block(const sw_ctx* ctx, const WfKernel& k) {
    return ctx->cell == kCellWide ? k.block : k.narrow_block;
}

int plain_occupancy(sw_ctx* ctx, const WfKernel& k, int qlen) {
    return kernel_occupancy(ctx, k, 0, qlen);
}

// Query rows one launch of a shape scores: the whole query when its profile
// fits one block, else the most whole passes whose profile does (a longer
// query is scored in row segments by consecutive launches that hand the
// boundary row on); 0 when not even one pass fits.
int launch_rows(sw_ctx* ctx, const WfKernel& k, int qlen) {
    if (plain_occupancy(ctx, k, qlen) > 0) return qlen;
    const int rows_pass = k.T * k.R;
    int p = 0;
    while ((int64_t)(p + 1) * rows_pass < qlen && plain_occupancy(ctx, k, (p + 1) * rows_pass) > 0)
        ++p;
    return p * rows_pass;
}

// Sum over the pairs [b, e) of max(ncols, m): the column steps of one pass
// whose segments last at least m steps.  Pairs are sorted by ncols
// descending, so the pairs below m are a suffix of the range.
double cols_at_least(const sw_ctx* ctx, int64_t b, int64_t e, uint32_t m) {
    const auto first = ctx->pair_ncols.begin();
    const int64_t i = std::partition_point(first + b, first + e,
                                           [m](uint32_t n) { return n >= m; }) - first;
    return (double)(ctx->pair_prefix[i] - ctx->pair_prefix[b]) + (double)m * (double)(e - i);
}

// Modelled cost of running pairs [b, e) with a shape, for contexts without a
// shape table entry that fits: thread steps x (R + 12.9) plus 25 per pass
// column and group, over an efficiency by group width (several groups in a
// warp diverge at their pair switches) and by resident warps.  The constants
// were fitted to the sweep of every compiled shape at 20 query lengths on a
// B200 (570,200 records); the model's pick is within 0.93 of the best shape
// on average there.  Columns per pass are counted as the streaming loop runs
// them: at least 2T + 2 steps for a pass a later pass depends on, 3 otherwise.
double shape_cost(sw_ctx* ctx, const WfKernel& k, int qlen, int64_t b, int64_t e) {
    const int rows = launch_rows(ctx, k, qlen);
    const int occ = rows > 0 ? plain_occupancy(ctx, k, rows) : 0;
    if (occ == 0 || e <= b) return occ == 0 ? 1e300 : 0.0;
    const double P = (qlen + k.T * k.R - 1) / (k.T * k.R);
    const double cols = (P - 1) * cols_at_least(ctx, b, e, 2 * k.T + 2) + cols_at_least(ctx, b, e, 3);
    const double work = cols * (k.T * (k.R + 12.9) + 25.1);
    const double g_width = k.T >= 32 ? 1.0 : k.T >= 16 ? 0.854 : k.T >= 8 ? 0.687 : 0.663;
    const double warps = (double)occ * plain_block(ctx, k) / 32.0;
    const double g_warps = warps < 12 ? 0.912 : warps < 20 ? 1.0 : 1.09;
    return work / (g_width * g_warps);
}

// The shape-table entry for a query length whose shapes fit it, or null (no
// table, no entry, a shape override, or the entry's shapes do not fit).
const sw_tuning_entry* find_entry(sw_ctx* ctx, int qlen) {
    if (ctx->has_override) return nullptr;
    for (const sw_tuning_entry& e : ctx->tuning) {
        if ((uint32_t)qlen > e.max_qlen) continue;
        const WfKernel* kl = find_kernel(e.cfg.long_group_width, e.cfg.long_rows_per_thread);
        const WfKernel* ks = find_kernel(e.cfg.short_group_width, e.cfg.short_rows_per_thread);
        if (kl && ks && plain_occupancy(ctx, *kl, qlen) > 0 && plain_occupancy(ctx, *ks, qlen) > 0)
            return &e;
        return nullptr;   // the tuned shape does not fit this length: the model chooses
    }
    return nullptr;
}

sw_kernel_config choose_config(sw_ctx* ctx, int qlen) {
    if (ctx->has_override) return ctx->override_cfg;
    if (const sw_tuning_entry* e = find_entry(ctx, qlen)) return e->cfg;
    int n = 0;
    const WfKernel* ks = wf_kernels(&n);
    const int64_t np = ctx->n_pairs;
    double best = 1e301;
    sw_kernel_config cfg{32, 32, 32, 32, 0};
    for (int i = 0; i < n; ++i) {
        const double c = shape_cost(ctx, ks[i], qlen, 0, np);
        if (c < best) {
            best = c;
            cfg = sw_kernel_config{ks[i].T, ks[i].R, ks[i].T, ks[i].R, 0};
        }
    }
    return cfg;
}

}  // namespace swb

extern "C" sw_status sw_set_kernel_config(sw_ctx* ctx, const sw_kernel_config* cfg) {
    if (!ctx) return SW_ERR_INVALID;
    if (!cfg) {
        ctx->has_override = false;
        return SW_OK;
    }
    if (!find_kernel(cfg->long_group_width, cfg->long_rows_per_thread) ||
        !find_kernel(cfg->short_group_width, cfg->short_rows_per_thread) || cfg->cutover < 0)
        SW_SET(ctx, SW_ERR_INVALID, "no compiled kernel for shape %dx%d / %dx%d",
               cfg->long_group_width, cfg->long_rows_per_thread, cfg->short_group_width,
               cfg->short_rows_per_thread);
    ctx->override_cfg = *cfg;
    ctx->has_override = true;
    return SW_OK;
}

extern "C" sw_status sw_set_tuning(sw_ctx* ctx, const sw_tuning_entry* entries, uint32_t n) {
    if (!ctx || (n && !entries)) return SW_ERR_INVALID;
    std::vector<sw_tuning_entry> tab(entries, entries + n);
    for (const sw_tuning_entry& e : tab) {
        if (!find_kernel(e.cfg.long_group_width, e.cfg.long_rows_per_thread) ||
            !find_kernel(e.cfg.short_group_width, e.cfg.short_rows_per_thread) || e.cfg.cutover < 0)
            SW_SET(ctx, SW_ERR_INVALID, "tuning entry names an uncompiled shape");
        for (const sw_plan_step& s : e.plan) {
            if (s.group_width == 0) break;
            if (!find_kernel(s.group_width, s.rows_per_thread) || s.passes < 0 ||
                s.passes > (1 << 20))
                SW_SET(ctx, SW_ERR_INVALID, "plan step %dx%d x %d passes: no such shape",
                       s.group_width, s.rows_per_thread, s.passes);
        }
    }
    for (size_t i = 1; i < tab.size(); ++i)
        if (tab[i].max_qlen < tab[i - 1].max_qlen)
            SW_SET(ctx, SW_ERR_INVALID, "tuning entries not sorted by max_qlen");
    ctx->tuning = std::move(tab);
    ctx->tuning_builtin = false;
    return SW_OK;
}

extern "C" sw_status sw_get_kernel_config(sw_ctx* ctx, uint32_t qlen, sw_kernel_config* cfg) {
    if (!ctx || !cfg) return SW_ERR_INVALID;
    if (!ctx->db_loaded) SW_SET(ctx, SW_ERR_STATE, "no DB loaded");
    *cfg = choose_config(ctx, (int)std::max<uint32_t>(qlen, 1));
    // the time model takes the place of the built-in table's cut-overs
    if (!ctx->has_override && ctx->tuning_builtin) cfg->cutover = 0;
    return SW_OK;
}

namespace swb {
sw_status describe_plan(sw_ctx* ctx, int qlen, sw_plan_step* steps, uint32_t capacity,
                        uint32_t* n_steps);
}

extern "C" sw_status sw_get_plan(sw_ctx* ctx, uint32_t qlen, sw_plan_step* steps,
                                 uint32_t capacity, uint32_t* n_steps) {
    if (!ctx || !n_steps || (capacity && !steps)) return SW_ERR_INVALID;
    if (!ctx->db_loaded) SW_SET(ctx, SW_ERR_STATE, "no DB loaded");
    if (qlen > kMaxQueryResidues)
        SW_SET(ctx, SW_ERR_UNSUPPORTED, "query of %u residues (at most %u)", qlen, kMaxQueryResidues);
    return describe_plan(ctx, (int)std::max<uint32_t>(qlen, 1), steps, capacity, n_steps);
}

extern "C" sw_status sw_get_shapes(int32_t* group_width, int32_t* rows_per_thread,
                                   int32_t* threads_per_block, uint32_t capacity,
                                   uint32_t* n_shapes) {
    if (!n_shapes) return SW_ERR_INVALID;
    int n = 0;
    const WfKernel* k = wf_kernels(&n);
    *n_shapes = (uint32_t)n;
    for (uint32_t i = 0; i < capacity && i < (uint32_t)n; ++i) {
        if (group_width) group_width[i] = k[i].T;
        if (rows_per_thread) rows_per_thread[i] = k[i].R;
        if (threads_per_block) threads_per_block[i] = k[i].block;
    }
    return SW_OK;
}

extern "C" sw_status sw_get_run_stats(const sw_ctx* ctx, sw_run_stats* out) {
    if (!ctx || !out) return SW_ERR_INVALID;
    *out = ctx->stats;
    return SW_OK;
}

// ---------------------------------------------------------------------------
// search
// ---------------------------------------------------------------------------

namespace swb {

// Enqueues the whole device sequence of one plain search on ctx->stream:
// first pass (one or two shapes), 32-bit re-score, top-k rounds.  The query
// must already be in d_query.  Returns the buffer holding the final k keys.
sw_status take_marks(sw_ctx* ctx, sw_ctx::Marks* m) {
    if (!ctx->spare.empty()) {
        *m = ctx->spare.back();
        ctx->spare.pop_back();
        return SW_OK;
    }
    for (auto& e : m->e) SW_CUDA(ctx, cudaEventCreate(&e));
    return SW_OK;
}

// A row segment of a plain search: the next `rows` query rows with shape k
// (consecutive launches of whole passes when the profile of all of them does
// not fit one block).
struct RowSeg {
    const WfKernel* k;
    int rows;
};
constexpr int kMaxRowSegs = SW_PLAN_STEPS + 1;

// Columns of one pass over the DB that an evenly loaded group of shape k gets.
double group_share(sw_ctx* ctx, const WfKernel& k, int qlen) {
    const int occ = std::max(1, plain_occupancy(ctx, k, qlen));
    const double groups = (double)occ * ctx->num_sms * (plain_block(ctx, k) / k.T);
    return (double)ctx->pair_cols_total / groups;
}

// The share a plan's steps are checked against: the one at the shape's nominal
// block size (sw_get_shapes), which the autotuner plans with.
double plan_share(sw_ctx* ctx, const WfKernel& k, int qlen) {
    const int occ = std::max(1, shape_occupancy(ctx, k, qlen));
    return (double)ctx->pair_cols_total / ((double)occ * ctx->num_sms * (k.block / k.T));
}

// Cut-over for a configuration without one: a DB whose longest pair needs more
// column steps than an evenly loaded bulk group gets (the bulk launch would end
// on a few serial chains: groups claim pairs longest first, so below that the
// long pairs finish inside the share) sends the pairs above a quarter of the
// share to the long-pair kernel; otherwise no split.
int auto_cutover(sw_ctx* ctx, const sw_kernel_config& cfg, int qlen) {
    if (ctx->n_pairs == 0) return 0;
    const WfKernel* k = find_kernel(cfg.short_group_width, cfg.short_rows_per_thread);
    if (!k) return 0;
    const double share = group_share(ctx, *k, qlen);
    if ((double)ctx->pair_ncols[0] <= share) return 0;
    return std::max(1024, (int)(share / 4));
}

// The row segments a plain search runs on its bulk pairs (the longest unit of
// them, a pair or a window, has `longest` columns; 0: there are none):
// the table entry's plan when it applies, else the whole query with the bulk
// shape ks (which also takes the rest of a plan without a rest step).  The
// plan is dropped (one segment) when a step names an uncompiled shape, when
// its fixed steps need more rows than the query has, when a segment's profile
// does not fit one pass in shared memory, or when a segment's shape is narrow
// enough that one group's even share of the columns is below the longest
// pair's (its launch would end on that pair's serial column steps: narrow
// shapes only pay with the long-pair split).
int build_plan(sw_ctx* ctx, int qlen, const WfKernel* ks, double longest, RowSeg* out) {
    out[0] = RowSeg{ks, qlen};
    const sw_tuning_entry* e = find_entry(ctx, qlen);
    if (!e || e->plan[0].group_width == 0 || !ks || longest <= 0) return 1;
    RowSeg segs[kMaxRowSegs];
    int n = 0, left = qlen;
    for (int i = 0; i < SW_PLAN_STEPS && left > 0; ++i) {
        const sw_plan_step& s = e->plan[i];
        if (s.group_width == 0) break;
        const WfKernel* k = find_kernel(s.group_width, s.rows_per_thread);
        if (!k || s.passes < 0) return 1;
        if (s.passes == 0) {
            segs[n++] = RowSeg{k, left};
            left = 0;
            break;
        }
        const int64_t rows = (int64_t)s.passes * k->T * k->R;
        if (rows > left) return 1;
        segs[n++] = RowSeg{k, (int)rows};
        left -= (int)rows;
    }
    if (left > 0) segs[n++] = RowSeg{ks, left};
    for (int i = 0; i < n; ++i)
        if (launch_rows(ctx, *segs[i].k, segs[i].rows) == 0 ||
            longest > plan_share(ctx, *segs[i].k, segs[i].rows))
            return 1;
    std::copy(segs, segs + n, out);
    return n;
}

// Pipelines of P warps one block of a long kernel holds (0: none fits).
int long_pipelines(sw_ctx* ctx, const LongKernel& k, int P, size_t* smem) {
    if (P > kLongMaxPasses) return 0;
    int n = 0;
    const sw_ctx::LongFit& f = ctx->long_fit[&k - long_kernels(&n)];
    const size_t dyn = (size_t)f.max_dyn;
    const int warp_regs = (f.regs + 7) / 8 * 8 * 32;
    int G = std::min(k.max_threads / 32, ctx->regs_per_sm / std::max(warp_regs, 1)) / P;
    while (G > 0 && k.smem(P, G) > dyn) --G;
    *smem = dyn;
    return G;
}

// The long-pair kernel for a query: the configured long shape when the
// configuration names one apart from the bulk shape (a shape table names one
// shape for both) and it is a compiled sw_long row count (group width 32)
// whose passes fit one pipeline, else the smallest row count that needs at most 3 passes (measured on B200:
// 2-3 passes per pair balance pipeline parallelism against per-step
// overhead), else at most kLongMaxPasses.  A block takes a whole SM:
// *pipelines is how many pipelines of *passes warps fit its registers and
// shared memory.  Returns null when nothing fits.
const LongKernel* choose_long(sw_ctx* ctx, const sw_kernel_config& cfg, int qlen, int* passes,
                              int* pipelines, size_t* smem_bytes) {
    int n = 0;
    const LongKernel* lk = long_kernels(&n);
    auto fits = [&](const LongKernel& k) {
        const int P = (qlen + 32 * k.R - 1) / (32 * k.R);
        size_t dyn = 0;
        const int G = long_pipelines(ctx, k, P, &dyn);
        if (G == 0) return false;
        *passes = P;
        *pipelines = G;
        *smem_bytes = dyn;
        return true;
    };
    const bool named = cfg.long_group_width != cfg.short_group_width ||
                       cfg.long_rows_per_thread != cfg.short_rows_per_thread;
    if (named && cfg.long_group_width == 32)
        for (int i = 0; i < n; ++i)
            if (lk[i].R == cfg.long_rows_per_thread && fits(lk[i])) return &lk[i];
    for (int i = 0; i < n; ++i)
        if ((qlen + 32 * lk[i].R - 1) / (32 * lk[i].R) <= 3 && fits(lk[i])) return &lk[i];
    for (int i = 0; i < n; ++i)
        if (fits(lk[i])) return &lk[i];
    return nullptr;
}

// The columns an alignment that scores above 0 can span: its gap costs stay
// below best_sum, the sum of its rows' best scores (each run of g residues
// costs gap_open + g * gap_extend), and at most qlen columns are matched.
// 0: no bound (free gap extension).
int64_t span_bound(const sw_ctx* ctx, int64_t qlen, int64_t best_sum) {
    if (ctx->params.gap_extend == 0) return 0;
    return qlen + std::max<int64_t>(0, best_sum - 1 - ctx->params.gap_open) / ctx->params.gap_extend;
}

// Windows of the pairs longer than `len` columns (0 windows: none are cut).
struct Windows {
    int len = 0, stride = 0;
    int64_t n_pairs = 0;     // pairs [0, n_pairs) are cut
    int n = 0;               // windows
};

// Pairs of more than `cols` columns: [0, pairs_above).
int64_t pairs_above(const sw_ctx* ctx, int64_t cols) {
    return std::partition_point(ctx->pair_ncols.begin(), ctx->pair_ncols.end(),
                                [cols](uint32_t n) { return (int64_t)n > cols; }) -
           ctx->pair_ncols.begin();
}

// Whether the windows of pairs [0, n_w) fit `units` of room; *windows: about
// how many there are (each pair's last partial stride as half a window, at
// most one).
bool windows_fit(const sw_ctx* ctx, int64_t n_w, int64_t len, int64_t stride, uint64_t units,
                 double* windows) {
    const double strides = ((double)ctx->pair_prefix[n_w] - (double)n_w * len) / stride;
    const double most = 2.0 * n_w + strides;
    *windows = 1.5 * n_w + strides;
    return most <= ctx->win_cap && most * (len / 8) <= (double)units;
}

void count_windows(const sw_ctx* ctx, Windows* w) {
    w->n = 0;
    for (int64_t p = 0; p < w->n_pairs; ++p)
        w->n += window_count((int)ctx->pair_ncols[p], w->len, w->stride);
}

// Windows for a bulk launch whose evenly loaded group gets `share` columns,
// with alignments spanning at most `span` columns.  A unit's columns are
// serial, so the launch lasts about max(share, longest unit) plus the tail of
// the last claims (a quarter of a unit); overlaps add columns to all groups.
// The window length with the least such estimate is taken, if that comes
// within 1.6 times the share (beyond that the long-pair kernel does better: on a
// DB with 43 % of its columns in long pairs, query 1,900, 5.2 ms against 40).
Windows plan_windows(const sw_ctx* ctx, double share, int64_t span) {
    Windows best;
    if (span <= 0 || ctx->n_pairs == 0 || (double)ctx->pair_ncols[0] <= 0.9 * share) return best;
    const double total = (double)ctx->pair_cols_total;
    double best_est = 1.6 * share;
    for (const double f : {1.0, 0.8, 0.65, 0.5, 0.4, 0.3, 0.2, 0.12}) {
        const int64_t len = (int64_t)(f * share) / 8 * 8;
        const int64_t stride = (len - span + 1) / 8 * 8;
        if (len < kMinWindow || stride < 64) break;
        if (len >= (int64_t)ctx->pair_ncols[0]) continue;
        const int64_t n_w = pairs_above(ctx, len);
        if (n_w > 3000) break;      // shorter windows only cut more pairs
        double windows = 0;
        if (!windows_fit(ctx, n_w, len, stride, ctx->win_units, &windows)) continue;
        const double extra = windows * len - (double)ctx->pair_prefix[n_w];
        const double est = share * (1.0 + extra / total) + 0.25 * len;
        if (est < best_est) {
            best_est = est;
            best.len = (int)len;
            best.stride = (int)stride;
            best.n_pairs = n_w;
        }
    }
    count_windows(ctx, &best);
    return best;
}

// ---- time model ----------------------------------------------------------
// Clocks of a first pass, for choosing between bulk shapes, windows and the
// long-pair kernel.  A column step of a thread's R rows is bound by the ALU
// pipe when an SM is full and by its own latency when few warps are on it;
// the constants were fitted to the kernels' measured rates on a B200 (bulk:
// 4.5 / 5.4 / 6.0 / 6.2 TCUPS at 8 / 16 / 24 / 48 rows on 350-residue records;
// long-pair kernel, clocks a step at 4 / 8 / 12 / 16 / 24 rows: 133 / 171 / 220 /
// 251 / 347 with one warp per scheduler, 185 / 263 / 356 / 422 / 612 with two,
// 306 / 494 / 653 / 815 / - with four).  Over 25 queries of 43..5,478 residues and
// DBs of 190..150,000 records the time it gives for the layout it picks came
// within 10 % of the measured one for all but a few launches under 0.15 ms.

// Cells an SM full of bulk groups of R rows per thread updates per clock.
double bulk_rate(int R) { return 24.0 * R / (R + 4.3); }

// Bulk launch over `units` units (pairs or windows, `cols` columns in all, the
// longest `longest`) in P passes on sms SMs.
double bulk_clocks(const WfKernel& k, int block, double P, double units, double cols,
                   double longest, double sms) {
    if (units <= 0) return 0.0;
    const double per_warp = 32.0 / k.T;
    const double warps = std::min(block / 32.0, std::max(1.0, units / per_warp / sms));
    const double step = std::max(60.0 + 11.7 * k.R, warps * 64.0 * k.R / bulk_rate(k.R));
    const double switches = units * (0.25 * (2 * k.T + 9));     // event steps per segment
    const double avg = (cols + switches) / (sms * warps * per_warp);
    // Units are claimed longest first, so the launch ends on short ones; but
    // warps of an SM differ in speed, so a unit as long as the even share ends
    // late (query 1,434 against 570,000 records, 4x40: 44.7 ms with units of up
    // to 0.56 of the share, 47.1 with 0.90, 48.1 with 0.95).
    const double tail = 0.15 * std::min({avg, longest, 2.0 * cols / units});
    return P * step * (std::max(avg, 1.18 * longest) + tail) + 15e3;
}

// The shape of a tall query's stack in a batch, whose pairs are [first, n_pairs).
// The built-in table and the cost model are for the plain kernel with its windows
// and long-pair split, which the stacked kernel has not; here the shape with the
// least time is taken, its longest pair's serial columns included (24 queries of
// 50..3,000 residues in 8x32 stacks of 1,024 rows against 60,000 records, 20 of
// them of 10,000..35,000 residues: 1,049 ms with the table's shapes, 213 with
// these; counting the chain of only one stack in full: 42 against 34 ms for 8
// queries of 2,000..3,000 and 20,000 records).
sw_kernel_config choose_stack_config(sw_ctx* ctx, int qlen, int64_t first) {
    if (ctx->has_override || first >= ctx->n_pairs ||
        (!ctx->tuning_builtin && find_entry(ctx, qlen)))
        return choose_config(ctx, qlen);      // the caller's shape
    const double cols = (double)(ctx->pair_cols_total - ctx->pair_prefix[first]);
    double best = 1e300;
    sw_kernel_config cfg = choose_config(ctx, qlen);
    int n = 0;
    const WfKernel* ks = wf_kernels(&n);
    for (int i = 0; i < n; ++i) {
        const WfKernel& k = ks[i];
        if (shape_occupancy(ctx, k, qlen) == 0) continue;
        const double t = bulk_clocks(k, k.block, (qlen + k.T * k.R - 1) / (k.T * k.R),
                                     (double)(ctx->n_pairs - first), cols,
                                     (double)ctx->pair_ncols[first], ctx->num_sms);
        if (t < best) {
            best = t;
            cfg = sw_kernel_config{k.T, k.R, k.T, k.R, 0};
        }
    }
    return cfg;
}

// One column step of the long-pair kernel with `warps` warps per SM.
double long_step_clocks(int R, int warps) {
    const int n = (warps + 3) / 4;      // warps per scheduler
    return std::max(90.0 + 10.8 * R, n * (36.0 + 10.6 * R) + (n == 2 ? 20.0 : 0.0));
}

double long_clocks(int R, int passes, int pipes, double pairs, double cols, double longest,
                   double sms) {
    const double step = 1.04 * long_step_clocks(R, passes * pipes);
    const double fill = (passes - 1) * 64.0 + 48.0;
    const double even = (cols + pairs * fill) / (sms * pipes);
    return step * (std::max(even, longest + fill) + (pairs > sms * pipes ? 0.3 * even * sms * pipes / pairs : 0.0)) +
           15e3;
}

// A long-pair split chosen by the model: pairs [0, n_long) to the long-pair
// kernel on `sms` SMs (`pipes` pipelines of `passes` warps each), the others
// to the bulk shape kb.
struct Split {
    const WfKernel* kb = nullptr;
    const LongKernel* lk = nullptr;
    int64_t n_long = 0;
    int passes = 0, pipes = 0, sms = 0;
    size_t smem = 0;
    bool join = false;
    Windows win;                // of the longest of those pairs (n 0: none)
    double clocks = 1e300;
};

// Bulk shapes the model chooses from: `given`, and (unless they are fixed) the
// two of each group width that suit the query's rows best.  A table's shape is
// tuned for a large DB; a small one, or one with long records, wants wider
// groups, whose units are fewer.
constexpr int kModelShapes = 16;
int model_shapes(sw_ctx* ctx, int qlen, const WfKernel* given, const WfKernel** shapes) {
    int n_shapes = 0;
    auto add = [&](const WfKernel* k) {
        if (!k || n_shapes == kModelShapes || launch_rows(ctx, *k, qlen) != qlen) return;
        for (int i = 0; i < n_shapes; ++i)
            if (shapes[i] == k) return;
        shapes[n_shapes++] = k;
    };
    add(given);
    const sw_tuning_entry* entry = find_entry(ctx, qlen);
    // a plan's shapes stay, and so does a shape from a caller's table
    const bool fixed = entry && (entry->plan[0].group_width != 0 || !ctx->tuning_builtin);
    int n_all = 0;
    const WfKernel* all = wf_kernels(&n_all);
    for (const int T : {32, 16, 8, 4}) {
        // the two row counts with the least time for the rows they compute
        const WfKernel* k2[2] = {nullptr, nullptr};
        double t2[2] = {1e300, 1e300};
        for (int i = 0; i < n_all && !fixed; ++i) {
            if (all[i].T != T) continue;
            const int rows = T * all[i].R;
            const double t = (qlen + rows - 1) / rows * (double)rows / bulk_rate(all[i].R);
            const int at = t < t2[0] ? 0 : t < t2[1] ? 1 : 2;
            if (at == 2) continue;
            if (at == 0) {
                k2[1] = k2[0];
                t2[1] = t2[0];
            }
            k2[at] = &all[i];
            t2[at] = t;
        }
        add(k2[0]);
        add(k2[1]);
    }
    return n_shapes;
}

constexpr int kModelLongs = 12;     // >= the compiled long-pair row counts

// The best split over cut-overs (every 1.5x in columns, down to every pair),
// row counts, SM shares, bulk shapes and windows of the longest pairs
// (alignments span at most `span` columns).
Split plan_split(sw_ctx* ctx, int qlen, int64_t span, const WfKernel* const* shapes,
                 int n_shapes) {
    Split best;
    const int64_t np = ctx->n_pairs;
    if (np == 0 || n_shapes == 0) return best;    // (no bulk shape: a query of row segments)
    struct Long {
        const LongKernel* k;
        int P, G;
        size_t smem;
    } longs[kModelLongs];
    int n_longs = 0, n_lk = 0;
    const LongKernel* lks = long_kernels(&n_lk);
    for (int i = 0; i < n_lk; ++i) {
        Long l{&lks[i], (qlen + 32 * lks[i].R - 1) / (32 * lks[i].R), 0, 0};
        l.G = long_pipelines(ctx, lks[i], l.P, &l.smem);
        if (l.G > 0 && n_longs < kModelLongs) longs[n_longs++] = l;
    }
    if (n_longs == 0) return best;
    const double total = (double)ctx->pair_cols_total;
    const int sms = ctx->num_sms;
    // Pairs [0, n_long) to the long-pair kernel as `units` units of `cols`
    // columns in all, the longest `longest`: more SMs for them end their launch
    // earlier and the bulk one later, so the best number of SMs is the first at
    // which theirs is done first, or the one before it.
    static constexpr int kSms[] = {1, 2, 4, 8, 12, 16, 24, 32, 48, 64, 96, 128};
    constexpr int kNumSms = sizeof(kSms) / sizeof(kSms[0]);
    auto consider = [&](int64_t n_long, double units, double cols, double longest,
                        const Windows* win) {
        // (no row count's step is shorter than the first's)
        if (longest * long_step_clocks(longs[0].k->R, 1) >= best.clocks) return;
        const double bulk_cols = total - (double)ctx->pair_prefix[n_long];
        auto at = [&](int on) {
            double tl = 1e300;
            const Long* l = nullptr;
            int pipes = 0;
            for (int i = 0; i < n_longs; ++i)
                for (int G = 1; G <= longs[i].G && (G - 1.0) * on < units; G *= 2) {
                    const double t = long_clocks(longs[i].k->R, longs[i].P, G, units, cols, longest, on);
                    if (t < tl) {
                        tl = t;
                        l = &longs[i];
                        pipes = G;
                    }
                }
            double tb = n_long == np ? 0.0 : 1e300;
            const WfKernel* kb = n_long == np ? shapes[0] : nullptr;
            for (int i = 0; i < n_shapes && n_long < np; ++i) {
                const WfKernel& k = *shapes[i];
                const double P = (qlen + k.T * k.R - 1) / (k.T * k.R);
                const double t = bulk_clocks(k, plain_block(ctx, k), P, (double)(np - n_long), bulk_cols,
                                             ctx->pair_ncols[n_long], sms - on);
                if (t < tb) {
                    tb = t;
                    kb = &k;
                }
            }
            const double t = std::max(tl, tb) + (win ? 10e3 : 0.0);
            if (kb && t < best.clocks) {
                best = Split{kb, l->k, n_long, l->P, pipes, on, l->smem, tl < 0.8 * tb, Windows{}, t};
                if (win) best.win = *win;
            }
            return tl <= tb;
        };
        if (n_long == np) {
            at(sms);
            return;
        }
        int lo = 0, hi = kNumSms - 1;
        while (hi > 0 && kSms[hi] >= sms) --hi;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (at(kSms[mid])) hi = mid;
            else lo = mid + 1;
        }
        at(kSms[lo]);
    };
    const int64_t longest = ctx->pair_ncols[0];
    int64_t prev = -1;
    for (double cut = (double)longest * 0.98;; cut /= 1.5) {
        const int64_t n_long = pairs_above(ctx, cut < 100.0 ? 0 : (int64_t)cut);
        if (n_long != prev && n_long > 0)
            consider(n_long, (double)n_long, (double)ctx->pair_prefix[n_long], (double)longest, nullptr);
        prev = n_long;
        if (cut < 100.0) break;
    }
    // Windows of the longest pairs, where the split's long launch waits on the
    // serial columns of a few of them: query 43 against 45,000 records and 90 of
    // 10,000..35,000 residues 2,426 -> 442 us, query 198 against 6,200 and 12 of
    // them 2,300 -> 371, query 1,875 against 984 and one 3,883 -> 1,059 (plain
    // split -> windows), query 144 against 200 records of up to 1,400 179 -> 122.
    if (span <= 0 || !best.lk) return best;
    for (const double f : {0.7, 0.5, 0.35, 0.25, 0.17, 0.12, 0.08, 0.05, 0.035}) {
        Windows w;
        w.len = (int)(f * longest) / 8 * 8;
        w.stride = (int)std::max<int64_t>((w.len - span + 1) / 8 * 8, 0);
        if (w.len < kMinWindow || w.stride < std::max(64, w.len / 8)) break;
        w.n_pairs = pairs_above(ctx, w.len);
        if (w.n_pairs > 3000) break;
        double n = 0;
        if (!windows_fit(ctx, w.n_pairs, w.len, w.stride, ctx->long_win_units, &n)) continue;
        prev = -1;
        for (double cut = w.len; cut > 100.0 && cut > 0.2 * w.len; cut /= 1.5) {
            const int64_t n_long = pairs_above(ctx, (int64_t)cut);
            if (n_long != prev)
                consider(n_long, n + (double)(n_long - w.n_pairs),
                         n * w.len + (double)(ctx->pair_prefix[n_long] - ctx->pair_prefix[w.n_pairs]),
                         w.len, &w);
            prev = n_long;
        }
    }
    count_windows(ctx, &best.win);
    return best;
}

// ---- long pairs of a batch or a serving round -----------------------------
//
// A paired-query launch scores every record of every double stack, so a record
// whose columns exceed a group's share of its smallest launch holds the whole
// launch, once per segment level of the tall stacks (48 requests against 57,000
// records with 20 of 10,000..35,000 residues: 100 ms a round, 25 of them work).
// The pairs above a cut-over go to sw_long_items instead, beside the launches.

// Clocks of the paired launches on `sms` SMs, longest record `longest`.  While
// every group has work a group's step takes as long as the SM's groups at 21.5
// cells per clock; what is left of the longest record's chain then runs beside
// few others, nearer to a step's own latency.  The chains start with the launch
// where the long units are dealt first (dealt), else with each double stack, so
// that the last one's overlaps its own stack only.  Over 110 batches of 2..64
// queries against 2,000..57,000 records in four shapes, without items: 0.81..1.21
// of the measured time for 8 of 10.  With plan_long_items' choice by it (and what
// it weighs the items at) a batch took 1.036 of the best choice's time in the
// geometric mean and in 3 of the 110 over 1.02 of the time without items, 1.06
// at most.  (With the whole chain at full-load steps, as it was, 45 queries of
// 81..478 residues against 32,360 records took 28.0 ms at 32x32, 22 without items.)
static double qp_clocks(const std::vector<QpLoad>& loads, double cols, double longest,
                        const QpKernel& k, double sms, bool dealt) {
    const double groups = (double)k.block / k.T;
    const double step = groups * k.T * k.R * 2.0 / 21.5;
    const double full = dealt ? 0.3 : 0.6;
    const double few = std::min(step, full * step + (1.0 - full) * (60.0 + 11.7 * k.R));
    double t = 0;
    for (const QpLoad& l : loads) {
        const double even = l.sum_passes * 2.0 * cols / (groups * sms);
        const double beside = dealt ? even : even * l.max_passes / std::max(l.sum_passes, 1.0);
        t += even * step + std::max(0.0, l.max_passes * longest - beside) * few + 20e3;
    }
    return t;
}

LongItemPlan plan_long_items(sw_ctx* ctx, const std::vector<uint32_t>& qlen,
                             const std::vector<QpLoad>& loads, const QpKernel& k, double chunks,
                             int64_t given) {
    LongItemPlan plan;
    const int64_t np = ctx->n_pairs;
    if (np == 0) return plan;
    // a query's items: pipelines, clocks a step, steps besides the columns' (half
    // the pipeline's fill, whose steps have fewer warps)
    struct Query {
        uint32_t q;
        int G;
        double step, fill;
    };
    std::vector<Query> queries;
    for (uint32_t q = 0; q < (uint32_t)qlen.size(); ++q) {
        if (qlen[q] == 0) continue;
        if (qlen[q] > (uint32_t)kLongItemRows) return plan;     // too long for a block's warps
        const int R = long_item_rows((int)qlen[q]);
        const int P = (int)((qlen[q] + 32 * R - 1) / (32 * R)), G = kLongItemWarps / P;
        queries.push_back(Query{q, G, 1.04 * long_step_clocks(R, P * G), (P - 1) * 32.0 + 48.0});
    }
    if (queries.empty()) return plan;
    const double total = (double)ctx->pair_cols_total / chunks, longest = ctx->pair_ncols[0];
    const int sms = ctx->num_sms;
    if (given < 0) {
        // (less than a tenth is within the estimates' error)
        double best = 0.9 * qp_clocks(loads, total, longest, k, sms, true);
        int64_t prev = 0;
        for (double cut = longest * 0.95; cut >= 256.0; cut /= 1.4) {
            const int64_t n = std::partition_point(ctx->pair_ncols.begin(), ctx->pair_ncols.end(),
                                                   [cut](uint32_t c) { return c > cut; }) -
                              ctx->pair_ncols.begin();
            if (n == prev || n == np) continue;
            prev = n;
            if (n > 16384) break;
            const double cols = (double)ctx->pair_prefix[n];
            double work = 0, chain = 0;         // of all items, of the longest
            for (const Query& q : queries) {
                const double G = (double)std::min<int64_t>(q.G, n);
                work += q.step * (cols / G + q.fill * std::ceil(n / G));
                chain = std::max(chain, q.step * (longest + q.fill));
            }
            for (const int x : {2, 4, 8, 12, 16, 24, 32, 48, 64, 80, 96}) {
                if (x >= sms) break;
                const double tl =
                    std::max(chain, work / x) + 0.1 * std::min(chain, work / x);
                const double tb =
                    qp_clocks(loads, total - cols / chunks, ctx->pair_ncols[n], k, sms - x, false);
                if (std::max(tl, tb) < best) {
                    best = std::max(tl, tb);
                    plan.n_long = n;
                    plan.sms = x;
                }
            }
        }
    } else {
        plan.n_long = given;
    }
    if (plan.n_long == 0) return plan;
    struct Item {
        uint32_t q, pair;
        double t;
    };
    std::vector<Item> list;
    for (const Query& q : queries) {
        plan.smem = std::max(plan.smem, long_item_smem((int)qlen[q.q]));
        for (int64_t p = 0; p < plan.n_long; p += q.G)
            list.push_back(Item{q.q, (uint32_t)p, (ctx->pair_ncols[p] + q.fill) * q.step});
    }
    if (plan.smem > (size_t)ctx->max_smem - 1024) return LongItemPlan{};
    if (given > 0) {
        // the pairs are given: SMs in proportion to the work, the items' as their
        // blocks hold it (an item lasts as long as its first pair, however many of
        // its pipelines have one: by the pairs' columns alone 52 requests of 309..7,284
        // residues waited 16 ms for their items after 59 ms of a round's launches)
        double wl = 0;
        for (const Item& i : list) wl += i.t;
        const double wb = qp_clocks(loads, total, 0.0, k, 1.0, true);
        plan.sms = std::max(1, std::min(sms * 2 / 3, (int)std::lround(sms * wl / (wl + wb))));
    }
    std::stable_sort(list.begin(), list.end(),
                     [](const Item& x, const Item& y) { return x.t > y.t; });
    for (const Item& i : list) {
        plan.items.push_back(i.q);
        plan.items.push_back(i.pair);
    }
    return plan;
}

// The plan's launch, at most `sms` blocks.
sw_status launch_long_items(sw_ctx* ctx, cudaStream_t stream, const LongItemPlan& plan,
                            const uint2* d_items, int* d_counter, const uint8_t* d_queries,
                            const uint32_t* d_qoff, const uint32_t* d_qlens, int* d_scores,
                            int* d_ovf, int* d_ovf_count, int ovf_cap, uint32_t* launches) {
    const int n = (int)plan.count();
    if (n == 0) return SW_OK;
    LongItemArgs a;
    a.db = ctx->d_db;
    a.pairs = ctx->d_pairs;
    a.n_pairs = (int)plan.n_long;
    a.items = d_items;
    a.n_items = n;
    a.counter = d_counter;
    a.queries = d_queries;
    a.qoff = d_qoff;
    a.qlens = d_qlens;
    a.mat = ctx->d_mat;
    a.gap_oe = ctx->params.gap_open + ctx->params.gap_extend;
    a.gap_e = ctx->params.gap_extend;
    a.scores = d_scores;
    a.n_records = (int)ctx->n_records;
    a.ovf_list = d_ovf;
    a.ovf_count = d_ovf_count;
    a.ovf_thresh = 32767 - std::max(ctx->max_score, 1) + 1;
    a.ovf_cap = ovf_cap;
    void* args[] = {&a};
    SW_CUDA(ctx, cudaLaunchKernel(long_item_kernel().fn[ctx->cell],
                                  dim3((unsigned)std::min(n, plan.sms)), dim3(32 * kLongItemWarps),
                                  args, plan.smem, stream));
    ++*launches;
    return SW_OK;
}

// How a plain search of qlen divides the DB's pairs: all to one bulk shape; the
// long ones cut into windows; or the long ones, [0, n_long), to the long-pair
// kernel and the rest (if any) to the bulk shape.
struct SearchLayout {
    sw_kernel_config cfg;
    Windows win;                       // long pairs cut into windows, for the long-pair
                                       // kernel with a split, else for the bulk launches
    int cutover = 0;
    bool split = false;
    int64_t n_long = 0;                // pairs of the long-pair kernel (split only), the
                                       // first win.n_pairs of them as windows
    const LongKernel* lk = nullptr;
    int lpasses = 0, lpipes = 0, lsms = 0;
    bool join = false;                 // the long launch ends well before the bulk one
    size_t lsmem = 0;
    int bulk_T = 0, bulk_R = 0;        // the bulk launches' shape ...
    int64_t bulk_b = 0, bulk_e = 0;    // ... pairs (after the windows) ...
    double longest = 0;                // ... columns of the longest unit ...
    int bulk_counter = 0;              // ... and claim counter
};

// Without a configured shape or cut-over: the layout the time model prefers.
// Returns false when it keeps one bulk shape, the configuration's long one, for
// every pair (windows and splits take the short one; they are the same but in a
// caller's table).
bool model_layout(sw_ctx* ctx, int qlen, int64_t span, SearchLayout* L) {
    const sw_kernel_config& cfg = L->cfg;
    const WfKernel* kb = find_kernel(cfg.short_group_width, cfg.short_rows_per_thread);
    const WfKernel* k1 = find_kernel(cfg.long_group_width, cfg.long_rows_per_thread);
    if (!kb || !k1 || ctx->n_pairs == 0) return false;
    const int rows = std::min(qlen, launch_rows(ctx, *kb, qlen));
    const double share = group_share(ctx, *kb, rows);
    if ((double)ctx->pair_ncols[0] <= 0.9 * share) return false;
    const double np = (double)ctx->n_pairs, total = (double)ctx->pair_cols_total;
    auto passes = [qlen](const WfKernel& k) { return (double)((qlen + k.T * k.R - 1) / (k.T * k.R)); };
    const double whole = bulk_clocks(*k1, plain_block(ctx, *k1), passes(*k1), np, total,
                                     ctx->pair_ncols[0], ctx->num_sms);
    const WfKernel* shapes[kModelShapes];
    const int n_shapes = model_shapes(ctx, qlen, kb, shapes);
    double windowed = 1e300;
    Windows win;
    const WfKernel* kw = kb;
    for (int i = 0; i < n_shapes; ++i) {
        const WfKernel& k = *shapes[i];
        const Windows w = plan_windows(ctx, group_share(ctx, k, qlen), span);
        if (w.n == 0) continue;
        const double t = bulk_clocks(k, plain_block(ctx, k), passes(k), np - w.n_pairs + w.n,
                                     total + (double)w.n * w.len - (double)ctx->pair_prefix[w.n_pairs],
                                     w.len, ctx->num_sms) + 15e3;
        if (t < windowed) {
            windowed = t;
            win = w;
            kw = &k;
        }
    }
    const Split sp = plan_split(ctx, qlen, span, shapes, n_shapes);
    const double least = std::min({whole, windowed, sp.clocks});
    if (least == whole) return false;
    if (least == windowed) {
        L->win = win;
        L->bulk_T = kw->T;
        L->bulk_R = kw->R;
        L->bulk_b = win.n_pairs;
        L->longest = win.len;
    } else {
        L->split = true;
        L->win = sp.win;
        L->n_long = sp.n_long;
        L->lk = sp.lk;
        L->lpasses = sp.passes;
        L->lpipes = sp.pipes;
        L->lsms = sp.sms;
        L->lsmem = sp.smem;
        L->join = sp.join;
        L->bulk_T = sp.kb->T;
        L->bulk_R = sp.kb->R;
        L->bulk_b = sp.n_long;
        L->cutover = sp.n_long < ctx->n_pairs ? (int)ctx->pair_ncols[sp.n_long] : 1;
        L->longest = sp.n_long < ctx->n_pairs ? (double)ctx->pair_ncols[sp.n_long] : 0.0;
    }
    L->bulk_e = ctx->n_pairs;
    L->bulk_counter = 1;
    return true;
}

void layout_search(sw_ctx* ctx, int qlen, int64_t span, SearchLayout* L) {
    const sw_kernel_config& cfg = L->cfg = choose_config(ctx, qlen);
    // A cut-over of a caller's table counts where the pairs it leaves to the bulk
    // launch fit a group's even share (the rule of a plan's steps): measured on a
    // large DB, it has a small one wait for them (4x40 with a cut-over of 4,096,
    // query 1,434: 44.2 ms against 44.5 without on 570,200 records, but 20.3
    // against 6.2 on 60,020 and 11.6 against 1.0 on 6,000).
    const WfKernel* ks = find_kernel(cfg.short_group_width, cfg.short_rows_per_thread);
    const bool callers_cut =
        cfg.cutover > 0 && !ctx->tuning_builtin && ks &&
        (double)cfg.cutover <= plan_share(ctx, *ks, std::min(qlen, launch_rows(ctx, *ks, qlen)));
    if (!ctx->has_override && !callers_cut) {
        if (model_layout(ctx, qlen, span, L)) return;
        L->bulk_T = cfg.long_group_width;
        L->bulk_R = cfg.long_rows_per_thread;
        L->bulk_b = 0;
        L->bulk_e = ctx->n_pairs;
        L->longest = ctx->n_pairs > 0 ? (double)ctx->pair_ncols[0] : 0.0;
        return;
    }
    // a shape override, or a caller's table with a cut-over: that cut-over, or
    // windows or a cut-over for the shape
    const WfKernel* kb = find_kernel(cfg.short_group_width, cfg.short_rows_per_thread);
    if (kb && cfg.cutover == 0)
        L->win = plan_windows(ctx, group_share(ctx, *kb, std::min(qlen, launch_rows(ctx, *kb, qlen))),
                              span);
    if (L->win.n > 0) {
        L->bulk_T = cfg.short_group_width;
        L->bulk_R = cfg.short_rows_per_thread;
        L->bulk_b = L->win.n_pairs;
        L->bulk_e = ctx->n_pairs;
        L->longest = L->win.len;
        return;
    }
    L->cutover = cfg.cutover > 0 ? cfg.cutover : auto_cutover(ctx, cfg, qlen);
    int64_t n_long = ctx->n_pairs;
    if (L->cutover > 0) {
        n_long = 0;
        while (n_long < ctx->n_pairs && (int)ctx->pair_ncols[n_long] > L->cutover) ++n_long;
    }
    L->split = L->cutover > 0 && n_long > 0 && n_long < ctx->n_pairs;
    if (L->split) {
        L->lk = choose_long(ctx, cfg, qlen, &L->lpasses, &L->lpipes, &L->lsmem);
        if (!L->lk) L->split = false;      // no pipelined shape for this length
    }
    if (L->split || (n_long < ctx->n_pairs && L->cutover > 0)) {
        // the short shape: beside the long-pair kernel, or alone for every
        // pair when no pair is above the cut-over or no pipelined shape fits
        L->bulk_T = cfg.short_group_width;
        L->bulk_R = cfg.short_rows_per_thread;
        L->bulk_b = L->split ? n_long : 0;
        L->bulk_counter = 1;
    } else {
        L->bulk_T = cfg.long_group_width;
        L->bulk_R = cfg.long_rows_per_thread;
        L->bulk_b = 0;
        L->bulk_counter = 0;
    }
    L->bulk_e = ctx->n_pairs;
    L->n_long = L->split ? n_long : 0;
    if (L->split) {
        // SMs and pipelines a block for the long launch: the best of the model for
        // its pairs and row count beside this bulk shape.  Few pipelines step faster,
        // which a few much longer pairs want; when only more SMs could make them
        // few, the launch took 100 SMs and the bulk one waited (query 500 against
        // 60,020 records, first pass at 8x40 6.3 ms, 2.9 now; at 4x40 6.4, 3.2).
        double best = 1e300;
        const double cols = (double)ctx->pair_prefix[n_long];
        const int G0 = L->lpipes;
        for (int x = 1; x < ctx->num_sms; x += 1 + x / 8) {
            const int most = (int)std::min<int64_t>(G0, (n_long + x - 1) / x);
            double tl = 1e300;
            int G = 0;
            for (int g = 1; g <= most; g = g < most ? std::min(2 * g, most) : g + 1) {
                const double t = long_clocks(L->lk->R, L->lpasses, g, (double)n_long, cols,
                                             ctx->pair_ncols[0], x);
                if (t < tl) {
                    tl = t;
                    G = g;
                }
            }
            const WfKernel* k = find_kernel(L->bulk_T, L->bulk_R);
            const double P = k ? (qlen + k->T * k->R - 1) / (k->T * k->R) : 1;
            const double tb = k ? bulk_clocks(*k, plain_block(ctx, *k), P,
                                              (double)(ctx->n_pairs - n_long),
                                              (double)ctx->pair_cols_total - cols,
                                              ctx->pair_ncols[n_long], ctx->num_sms - x) : 0.0;
            const double t = std::max(tl, tb) + 0.01 * std::min(tl, tb);
            if (t < best) {
                best = t;
                L->lsms = x;
                L->lpipes = G;
            }
        }
    }
    L->longest = L->bulk_b < L->bulk_e ? (double)ctx->pair_ncols[L->bulk_b] : 0.0;
}

// span_bound for any query of a length.
int64_t length_span(const sw_ctx* ctx, int64_t qlen) {
    return span_bound(ctx, qlen, qlen * ctx->max_score);
}

// span_bound for a query whose residues the host holds.
int64_t query_span(const sw_ctx* ctx, const uint8_t* query, int64_t qlen) {
    int64_t sum = 0;
    for (int64_t i = 0; i < qlen; ++i) sum += ctx->row_best[query[i] & 31];
    return span_bound(ctx, qlen, sum);
}

// sw_get_plan: the row segments enqueue_search would run.
sw_status describe_plan(sw_ctx* ctx, int qlen, sw_plan_step* steps, uint32_t capacity,
                        uint32_t* n_steps) {
    SearchLayout L;
    layout_search(ctx, qlen, length_span(ctx, qlen), &L);
    const WfKernel* k = find_kernel(L.bulk_T, L.bulk_R);
    if (!k) SW_SET(ctx, SW_ERR_INVALID, "no kernel %dx%d", L.bulk_T, L.bulk_R);
    RowSeg plan[kMaxRowSegs];
    const int n = build_plan(ctx, qlen, k, L.longest, plan);
    *n_steps = (uint32_t)n;
    for (int i = 0; i < n && (uint32_t)i < capacity; ++i) {
        const int rp = plan[i].k->T * plan[i].k->R;
        steps[i] = sw_plan_step{plan[i].k->T, plan[i].k->R, (plan[i].rows + rp - 1) / rp};
    }
    return SW_OK;
}

sw_status enqueue_search(sw_ctx* ctx, const uint8_t* d_query, int qlen, int64_t span,
                         int32_t* d_scores_rec, unsigned long long** keys_final,
                         uint32_t* launches) {
    cudaStream_t st = ctx->stream;
    SearchLayout L;
    layout_search(ctx, qlen, span, &L);
    ctx->stats.used = L.cfg;
    ctx->stats.used.cutover = L.cutover;
    if (L.win.n > 0 && !L.split) {
        ctx->stats.used.short_group_width = ctx->stats.used.long_group_width = L.bulk_T;
        ctx->stats.used.short_rows_per_thread = ctx->stats.used.long_rows_per_thread = L.bulk_R;
    }
    *launches = 0;
    const bool split = L.split;
    const int64_t n_long = L.n_long;
    const LongKernel* lk = L.lk;
    const int lpasses = L.lpasses;
    const int lpipes = L.lpipes;
    if (split) {
        ctx->stats.used.short_group_width = L.bulk_T;
        ctx->stats.used.short_rows_per_thread = L.bulk_R;
        ctx->stats.used.long_group_width = 32;
        ctx->stats.used.long_rows_per_thread = lk->R;
    }
    const int ovf_thresh = 32767 - std::max(ctx->max_score, 1) + 1;
    // With a cut-over, the long pairs run concurrently on the side stream in
    // sw_long blocks (one warp per query pass, the passes of a pair pipelined
    // across warps, several pipelines per block, one block per SM) on SMs the
    // bulk grid leaves free (as many as the time model gives them).  The bulk
    // launches take the other pairs in the row segments of
    // the length's plan.
    RowSeg plan[kMaxRowSegs];
    int nplan = 0;
    // every shape is checked before anything is launched: a search refused
    // half-way would leave a launch in flight that writes into the next one
    const int bulk_win = split ? 0 : L.win.n;
    if (L.bulk_e > L.bulk_b || bulk_win > 0) {
        const WfKernel* k = find_kernel(L.bulk_T, L.bulk_R);
        if (!k) SW_SET(ctx, SW_ERR_INVALID, "no kernel %dx%d", L.bulk_T, L.bulk_R);
        if (launch_rows(ctx, *k, qlen) == 0)
            SW_SET(ctx, SW_ERR_UNSUPPORTED,
                   "one pass of shape %dx%d does not fit shared memory (profile %zu bytes)",
                   L.bulk_T, L.bulk_R, k->smem(L.bulk_T * L.bulk_R));
        nplan = build_plan(ctx, qlen, k, L.longest, plan);
        if (nplan > 1) {
            ctx->stats.used.short_group_width = plan[0].k->T;
            ctx->stats.used.short_rows_per_thread = plan[0].k->R;
        }
    }
    // the search's timing events, taken after every check (a refused search
    // holds none), then its buffers cleared
    sw_ctx::Marks mk{};
    sw_status ms = take_marks(ctx, &mk);
    if (ms != SW_OK) return ms;
    mk.fp_launches = 0;
    mk.cells = (uint64_t)qlen * ctx->n_residues;
    SW_CUDA(ctx, cudaEventRecord(mk.e[0], st));
    SW_CUDA(ctx, cudaMemsetAsync(ctx->d_counters, 0,
                                 (size_t)(kCounters + ctx->n_records + 1) * sizeof(int), st));
    SW_CUDA(ctx, cudaEventRecord(mk.e[1], st));
    if (L.win.n > 0) {
        WindowArgs w;
        w.db = ctx->d_db;
        w.pairs = ctx->d_pairs;
        w.len = L.win.len;
        w.stride = L.win.stride;
        w.base = (uint32_t)ctx->units;
        w.win_pairs = ctx->d_win_pairs;
        w.win_ids = ctx->d_win_ids;
        void* args[] = {&w};
        SW_CUDA(ctx, cudaLaunchKernel((const void*)sw_windows, dim3((unsigned)L.win.n_pairs),
                                      dim3(kWindowThreads), args, 0, st));
        ++*launches;
    }
    int reserved_sms = 0;
    if (split) {
        reserved_sms = L.lsms;
        SW_CUDA(ctx, cudaEventRecord(ctx->fork_ev, st));
        SW_CUDA(ctx, cudaStreamWaitEvent(ctx->side_stream, ctx->fork_ev, 0));
        LongArgs la;
        la.db = ctx->d_db;
        la.pairs = ctx->d_pairs;
        la.n_win = L.win.n;
        la.win_pairs = ctx->d_win_pairs;
        la.win_ids = ctx->d_win_ids;
        la.pair_begin = (int)L.win.n_pairs;
        la.count = L.win.n + (int)(n_long - L.win.n_pairs);
        la.counter = ctx->d_counters;      // counter 0: the long pairs' claims
        la.query = d_query;
        la.qlen = qlen;
        la.passes = lpasses;
        la.mat = ctx->d_mat;
        la.gap_oe = ctx->params.gap_open + ctx->params.gap_extend;
        la.gap_e = ctx->params.gap_extend;
        la.scores = ctx->d_scores;
        la.n_records = (int)ctx->n_records;
        la.ovf_list = ctx->d_ovf;
        la.ovf_count = ctx->d_counters + 2;
        la.ovf_thresh = ovf_thresh;
        la.ovf_cap = (int)ctx->n_records + 1;
        void* args[] = {&la};
        SW_CUDA(ctx, cudaEventRecord(mk.e[4], ctx->side_stream));
        SW_CUDA(ctx, cudaLaunchKernel(
                         lk->fn[ctx->cell],
                         dim3((unsigned)std::min<int64_t>(reserved_sms, (la.count + lpipes - 1) / lpipes)),
                         dim3(lpasses * lpipes * 32), args, L.lsmem, ctx->side_stream));
        SW_CUDA(ctx, cudaEventRecord(mk.e[5], ctx->side_stream));
        ++*launches;
        ++mk.fp_launches;
        SW_CUDA(ctx, cudaEventRecord(mk.e[6], st));
    }
    mk.split = split;
    // Row segments of the plan (one for most lengths), each in launches of
    // whole passes up to what one block's profile holds: every launch but the
    // first reads the boundary row the one before wrote (pass0 counts the
    // query's passes before it, whatever their shapes: the row holds one
    // 8-byte (H, F) entry per column and parity of the pass index, so its
    // layout does not depend on the shape), and scores merge by maximum.
    int r0 = 0, passes_before = 0;
    for (int pi = 0; pi < nplan; ++pi) {
        const WfKernel* k = plan[pi].k;
        const int seg_rows = launch_rows(ctx, *k, plan[pi].rows);
        for (int s0 = 0; s0 < plan[pi].rows; s0 += seg_rows) {
            const int rows = std::min(seg_rows, plan[pi].rows - s0);
            const int occ = plain_occupancy(ctx, *k, rows);
            if (r0 > 0)   // the previous launch has claimed every pair
                SW_CUDA(ctx, cudaMemsetAsync(ctx->d_counters + L.bulk_counter, 0, sizeof(int), st));
            WfArgs a;
            a.db = ctx->d_db;
            a.pairs = ctx->d_pairs;
            a.pair_begin = (int)L.bulk_b;
            a.pair_count = (int)(L.bulk_e - L.bulk_b) + bulk_win;
            a.win_pairs = ctx->d_win_pairs;
            a.win_ids = ctx->d_win_ids;
            a.n_win = bulk_win;
            a.query = d_query + r0;
            a.qlen = rows;
            a.pass0 = passes_before;
            a.more = r0 + rows < qlen ? 1 : 0;
            a.mat = ctx->d_mat;
            a.gap_oe = ctx->params.gap_open + ctx->params.gap_extend;
            a.gap_e = ctx->params.gap_extend;
            a.counter = ctx->d_counters + L.bulk_counter;
            a.bnd = ctx->d_bnd;
            a.scores = ctx->d_scores;
            a.n_records = (int)ctx->n_records;
            a.ovf_list = ctx->d_ovf;
            a.ovf_count = ctx->d_counters + 2;
            a.ovf_thresh = ovf_thresh;
            void* args[] = {&a};
            // The first launch leaves the long launch its SMs (blocks that
            // found them first would hold them to the end); a later row
            // segment's blocks wait for theirs.
            const bool first = r0 == 0;
            int64_t grid = (int64_t)occ * (ctx->num_sms - (first ? reserved_sms : 0));
            const int block = plain_block(ctx, *k);
            // a warp claims 32 / T pairs at a time: no more blocks than claims
            // (few pairs spread one warp per SM)
            const int64_t per_claim = 32 / k->T;
            grid = std::min<int64_t>(grid, (a.pair_count + per_claim - 1) / per_claim);
            grid = std::max<int64_t>(grid, 1);
            a.block0 = 0;
            a.first_blocks = (int)std::min<int64_t>(
                grid, std::max<int64_t>(1, (int64_t)occ * (ctx->num_sms - reserved_sms)));
            SW_CUDA(ctx, cudaLaunchKernel(k->fn[ctx->cell], dim3((unsigned)grid), dim3(block), args,
                                          k->smem(rows), st));
            ++*launches;
            ++mk.fp_launches;
            if (L.join && first && rows == qlen) {
                // the whole query in one launch: once the long pairs are done
                // their SMs take part in it
                a.block0 = a.first_blocks;
                SW_CUDA(ctx, cudaLaunchKernel(k->fn[ctx->cell], dim3((unsigned)(occ * reserved_sms)),
                                              dim3(block), args, k->smem(rows), ctx->side_stream));
                ++*launches;
                ++mk.fp_launches;
            }
            r0 += rows;
            passes_before += (rows + k->T * k->R - 1) / (k->T * k->R);
        }
    }
    if (split) {
        SW_CUDA(ctx, cudaEventRecord(mk.e[7], st));
        SW_CUDA(ctx, cudaEventRecord(ctx->join_ev, ctx->side_stream));
        SW_CUDA(ctx, cudaStreamWaitEvent(st, ctx->join_ev, 0));
    }
    SW_CUDA(ctx, cudaEventRecord(mk.e[2], st));
    {
        RescoreArgs r;
        r.db = ctx->d_db;
        r.pairs = ctx->d_pairs;
        r.query = d_query;
        r.qlen = qlen;
        r.mat = ctx->d_mat;
        r.gap_oe = ctx->params.gap_open + ctx->params.gap_extend;
        r.gap_e = ctx->params.gap_extend;
        r.queries = nullptr;
        r.qoff = nullptr;
        r.qlens = nullptr;
        r.n_records = (int)ctx->n_records;
        r.ovf_list = ctx->d_ovf;
        r.ovf_count = ctx->d_counters + 2;
        r.ovf_cap = (int)ctx->n_records + 1;
        r.scratch = ctx->d_rs_scratch;
        r.max_cols = ctx->max_cols;
        r.scores = ctx->d_scores;
        void* args[] = {&r};
        SW_CUDA(ctx, cudaLaunchKernel((const void*)sw_rescore32, dim3(kRescoreBlocks), dim3(64),
                                      args, 0, st));
        ++*launches;
    }
    // top-k rounds: n -> ceil(n/4096)*k -> ... -> k
    const int k = ctx->params.top_k;
    long long n = ctx->n_records;
    int buf = 0;
    const unsigned long long* keys_in = nullptr;
    bool first = true;
    while (true) {
        const long long blocks = std::max<long long>(1, (n + kTopkKeys - 1) / kTopkKeys);
        TopkArgs t;
        t.scores = ctx->d_scores;
        t.perm = ctx->d_perm;
        t.keys_in = first ? nullptr : keys_in;
        t.n = n;
        t.k = k;
        t.cap = (ctx->params.flags & SW_FLAG_REFERENCE_CAP) ? 1 : 0;
        t.scores_by_record = first ? d_scores_rec : nullptr;
        t.keys_out = ctx->d_keys[buf];
        t.in_stride = 0;
        t.rec_stride = 0;
        t.out_stride = 0;
        t.rows = nullptr;
        t.count = blocks == 1 ? ctx->d_counters + 2 : nullptr;
        void* args[] = {&t};
        SW_CUDA(ctx, cudaLaunchKernel((const void*)sw_topk_round, dim3((unsigned)blocks),
                                      dim3(kTopkThreads), args, 0, st));
        ++*launches;
        keys_in = ctx->d_keys[buf];
        buf ^= 1;
        first = false;
        if (blocks == 1) break;
        n = blocks * (long long)k;
    }
    *keys_final = const_cast<unsigned long long*>(keys_in);
    SW_CUDA(ctx, cudaEventRecord(mk.e[3], st));
    mk.launches = *launches;
    ctx->pending.push_back(mk);
    return SW_OK;
}

// Waits for the stream and folds the pending searches' event timings into
// the totals; returns the last search's (whole, first pass) device times.
sw_status drain(sw_ctx* ctx, float* last_ms, float* last_fp_ms) {
    SW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (auto& m : ctx->pending) {
        float whole = 0.f, fp = 0.f, lms = 0.f, bms = 0.f;
        SW_CUDA(ctx, cudaEventElapsedTime(&whole, m.e[0], m.e[3]));
        SW_CUDA(ctx, cudaEventElapsedTime(&fp, m.e[1], m.e[2]));
        if (m.split) {
            SW_CUDA(ctx, cudaEventElapsedTime(&lms, m.e[4], m.e[5]));
            SW_CUDA(ctx, cudaEventElapsedTime(&bms, m.e[6], m.e[7]));
        }
        ctx->stats.long_ms = lms;
        ctx->stats.bulk_ms = bms;
        ctx->totals.search_ms += whole;
        ctx->totals.first_pass_ms += fp;
        ctx->totals.first_pass_launches += m.fp_launches;
        ctx->totals.launches += m.launches;
        ctx->totals.cells += m.cells;
        ctx->totals.queries += 1;
        if (last_ms) *last_ms = whole;
        if (last_fp_ms) *last_fp_ms = fp;
        ctx->spare.push_back(m);
    }
    ctx->pending.clear();
    return SW_OK;
}

sw_status ensure_query_buffers(sw_ctx* ctx, size_t qlen) {
    if (qlen <= ctx->query_cap) return SW_OK;
    size_t cap = std::max<size_t>(qlen, 4096);
    dev_free(ctx->d_query);
    if (ctx->h_query) cudaFreeHost(ctx->h_query);
    ctx->h_query = nullptr;
    ctx->query_cap = 0;
    if (dev_alloc(&ctx->d_query, cap) != cudaSuccess) SW_SET(ctx, SW_ERR_NOMEM, "query buffer");
    if (cudaMallocHost((void**)&ctx->h_query, cap) != cudaSuccess)
        SW_SET(ctx, SW_ERR_NOMEM, "pinned query buffer");
    // (the keys, then the count of re-scored records)
    if (!ctx->h_keys && cudaMallocHost((void**)&ctx->h_keys,
                                       (kMaxTopK + 1) * sizeof(unsigned long long)) != cudaSuccess)
        SW_SET(ctx, SW_ERR_NOMEM, "pinned key buffer");
    ctx->query_cap = cap;
    return SW_OK;
}

}  // namespace swb

extern "C" sw_status sw_search(sw_ctx* ctx, const uint8_t* query, uint32_t qlen, sw_hit* hits,
                               uint32_t* n_hits, int32_t* scores) {
    if (!ctx) return SW_ERR_INVALID;
    if (ctx->serve) return SW_ERR_BUSY;   // the serving loop owns the stream and the DB
    return swb::search_host(ctx, query, qlen, hits, n_hits, scores);
}

namespace swb {

sw_status search_host(sw_ctx* ctx, const uint8_t* query, uint32_t qlen, sw_hit* hits,
                      uint32_t* n_hits, int32_t* scores) {
    if (!ctx->db_loaded) SW_SET(ctx, SW_ERR_STATE, "no DB loaded (call sw_db_load first)");
    if ((qlen && !query) || (!hits && ctx->params.top_k > 0) || !n_hits)
        SW_SET(ctx, SW_ERR_INVALID, "null argument");
    if (qlen > kMaxQueryResidues)
        SW_SET(ctx, SW_ERR_UNSUPPORTED, "query of %u residues (at most %u)", qlen, kMaxQueryResidues);
    const double t0 = now_ms();
    const int k = ctx->params.top_k;
    for (int i = 0; i < k; ++i) hits[i] = sw_hit{0, 0, 0};
    *n_hits = 0;
    ctx->stats = sw_run_stats{};
    if (qlen == 0 || ctx->n_records == 0) {
        if (scores) memset(scores, 0, (size_t)ctx->n_records * sizeof(int32_t));
        ctx->stats.total_ms = now_ms() - t0;
        return SW_OK;
    }
    for (uint32_t i = 0; i < qlen; ++i)
        if (query[i] > 24) SW_SET(ctx, SW_ERR_INVALID, "query code %d at %u", query[i], i);
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    sw_status st = ensure_query_buffers(ctx, qlen);
    if (st != SW_OK) return st;
    memcpy(ctx->h_query, query, qlen);
    SW_CUDA(ctx, cudaMemcpyAsync(ctx->d_query, ctx->h_query, qlen, cudaMemcpyHostToDevice,
                                 ctx->stream));
    unsigned long long* keys = nullptr;
    uint32_t launches = 0;
    st = enqueue_search(ctx, ctx->d_query, (int)qlen, query_span(ctx, query, qlen),
                        scores ? ctx->d_scores_rec : nullptr, &keys, &launches);
    if (st != SW_OK) return st;
    // the hits and, behind them, the count of re-scored records
    SW_CUDA(ctx, cudaMemcpyAsync(ctx->h_keys, keys, (size_t)(k + 1) * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToHost, ctx->stream));
    if (scores)
        SW_CUDA(ctx, cudaMemcpyAsync(scores, ctx->d_scores_rec,
                                     (size_t)ctx->n_records * sizeof(int32_t),
                                     cudaMemcpyDeviceToHost, ctx->stream));
    float kms = 0.f, fpms = 0.f;
    st = drain(ctx, &kms, &fpms);
    if (st != SW_OK) return st;
    SW_CUDA(ctx, cudaGetLastError());
    uint32_t m = 0;
    for (int i = 0; i < k; ++i) {
        const unsigned long long key = ctx->h_keys[i];
        if (key == 0ull) break;
        hits[m].score = (int32_t)(key >> 32);
        hits[m].reserved = 0;
        hits[m].index = 0xffffffffull - (key & 0xffffffffull);
        ++m;
    }
    *n_hits = m;
    ctx->stats.kernel_ms = kms;
    ctx->stats.first_pass_ms = fpms;
    ctx->stats.cells = (uint64_t)qlen * ctx->n_residues;
    ctx->stats.rescored = ctx->h_keys[k];
    ctx->stats.launches = launches;
    ctx->stats.queries = 1;
    ctx->stats.total_ms = now_ms() - t0;
    return SW_OK;
}

}  // namespace swb

extern "C" sw_status sw_search_device(sw_ctx* ctx, const uint8_t* d_query, uint32_t qlen,
                                      int32_t* d_scores) {
    if (!ctx) return SW_ERR_INVALID;
    if (ctx->serve) return SW_ERR_BUSY;   // the serving loop owns the stream and the DB
    if (!ctx->db_loaded) SW_SET(ctx, SW_ERR_STATE, "no DB loaded (call sw_db_load first)");
    if (!d_query || qlen == 0) SW_SET(ctx, SW_ERR_INVALID, "empty query");
    if (qlen > kMaxQueryResidues)
        SW_SET(ctx, SW_ERR_UNSUPPORTED, "query of %u residues (at most %u)", qlen, kMaxQueryResidues);
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    ctx->stats = sw_run_stats{};
    unsigned long long* keys = nullptr;
    uint32_t launches = 0;
    sw_status st = enqueue_search(ctx, d_query, (int)qlen, length_span(ctx, qlen), d_scores, &keys,
                                  &launches);
    if (st != SW_OK) return st;
    ctx->stats.cells = (uint64_t)qlen * ctx->n_residues;
    ctx->stats.launches = launches;
    ctx->stats.queries = 1;
    return SW_OK;
}

extern "C" sw_status sw_set_stream(sw_ctx* ctx, void* cuda_stream) {
    if (!ctx) return SW_ERR_INVALID;
    if (ctx->serve) return SW_ERR_BUSY;   // the serving loop owns the stream and the DB
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    sw_status st = drain(ctx, nullptr, nullptr);
    if (st != SW_OK) return st;
    ctx->stream = cuda_stream ? (cudaStream_t)cuda_stream : ctx->own_stream;
    return SW_OK;
}

extern "C" sw_status sw_sync(sw_ctx* ctx) {
    if (!ctx) return SW_ERR_INVALID;
    SW_CUDA(ctx, cudaSetDevice(ctx->device));
    sw_status st = drain(ctx, nullptr, nullptr);
    if (st != SW_OK) return st;
    SW_CUDA(ctx, cudaGetLastError());
    return SW_OK;
}

extern "C" sw_status sw_reset_totals(sw_ctx* ctx) {
    if (!ctx) return SW_ERR_INVALID;
    sw_status st = sw_sync(ctx);
    ctx->totals = sw_totals{};
    return st;
}

extern "C" sw_status sw_get_totals(const sw_ctx* ctx, sw_totals* out) {
    if (!ctx || !out) return SW_ERR_INVALID;
    *out = ctx->totals;
    return SW_OK;
}
