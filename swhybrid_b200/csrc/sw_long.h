// sw_long.h -- the long-pair first pass (sw_long.cu): arguments and the table
// of compiled row counts.
#pragma once
#include <cstddef>
#include <cstdint>

#include "sw_device.cuh"
#include "sw_registry.h"

namespace swb {

constexpr int kLongMaxPasses = 16;       // query passes of 32 x R rows = warps per pipeline
constexpr int kLongMaxWarps = 32;        // pipelines x passes per block

struct LongArgs {
    const uint4* db;            // pair column streams
    const Pair2* pairs;         // pair table, ncols descending
    int n_win;                  // units: n_win windows of long pairs (see sw_windows),
    const Pair2* win_pairs;     // ... table entries of their own
    const uint32_t* win_ids;    // ... and the pair each belongs to,
    int pair_begin;             // then the pairs [pair_begin, pair_begin + count - n_win)
    int count;
    int* counter;               // units claimed so far (one pipeline per unit)
    const uint8_t* query;
    int qlen;                   // at most kLongMaxPasses * 32 * R rows
    int passes;                 // ceil(qlen / (32 R)); blockDim.x = 32 * passes * pipelines
    const int8_t* mat;
    int gap_oe, gap_e;          // open + extend, extend
    int* scores;                // by sorted position
    int n_records;
    int* ovf_list;              // positions whose 16-bit lanes may have wrapped
    int* ovf_count;
    int ovf_thresh;
    int ovf_cap;
};

struct LongKernel {
    int R;                                      // query rows per thread; 32 threads per pass
    const void* fn[kPlainCells];                // __global__ sw_long<R, cell>
    size_t (*smem)(int passes, int pipelines);  // dynamic shared memory of one block
    int max_threads;                            // the kernel's launch bound
};

const LongKernel* long_kernels(int* n);

// Long pairs of several queries (batched search, serving): see sw_long_items.
constexpr int kLongItemWarps = 16;
constexpr int kLongItemRows = 32 * 16 * kLongItemWarps;    // longest query

// Query rows per lane: the least whose passes the block's warps hold.
__host__ __device__ constexpr int long_item_rows(int qlen) {
    return qlen <= 32 * 4 * kLongItemWarps ? 4 : qlen <= 32 * 8 * kLongItemWarps ? 8 : 16;
}

struct LongItemArgs {
    const uint4* db;
    const Pair2* pairs;         // the long pairs are [0, n_pairs), ncols descending
    int n_pairs;
    const uint2* items;         // (query, first pair), longest first
    int n_items;
    int* counter;               // items claimed so far
    const uint8_t* queries;     // query q: codes at queries + qoff[q], qlens[q] of them
    const uint32_t* qoff;
    const uint32_t* qlens;
    const int8_t* mat;
    int gap_oe, gap_e;
    int* scores;                // [query][sorted position]
    int n_records;
    int* ovf_list;              // query * n_records + position
    int* ovf_count;
    int ovf_thresh;
    int ovf_cap;
};

struct LongItemKernel {
    const void* fn[kPlainCells];                // __global__ sw_long_items<cell>
};

const LongItemKernel& long_item_kernel();
size_t long_item_smem(int qlen);                // dynamic shared memory of a query's items

}  // namespace swb
