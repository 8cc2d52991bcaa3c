// sw_registry.h -- table of compiled first-pass kernel shapes.
#pragma once
#include <cstddef>

namespace swb {

// Cell variants of the plain kernel (CellWide / CellNarrow, sw_wavefront.cuh),
// chosen per context by plain_cell() from the matrix and the gap costs.
enum PlainCell {
    kCellWide = 0,                 // any matrix
    kCellNarrow = 1,               // entries in [-q, 127 - q]: gap costs at run time ...
    kCellNarrow12_2 = 2,           // ... open+extend 12, extend 2 (the defaults, 10/2)
    kCellNarrow12_1 = 3,           // ... open+extend 12, extend 1 (11/1)
    kPlainCells = 4
};

struct WfKernel {
    int T;                         // threads per record pair
    int R;                         // query rows per thread
    int block;                     // threads per block (stacked kernel, plain with CellWide)
    int narrow_block;              // threads per block, plain with CellNarrow
    const void* fn[kPlainCells];   // __global__ sw_wavefront<T, R, ., cell> (plain)
    size_t (*smem)(int qlen);      // shared-memory bytes for a query length
    const void* batch_fn;          // __global__ sw_batch<T, R, block> (batched)
};

// All instantiated shapes (sw_wf_t*.cu).
const WfKernel* wf_kernels(int* n);

// Paired-query batched kernel shapes (sw_qp.cu).
struct QpKernel {
    int T, R, block;
    const void* fn[kPlainCells];   // __global__ sw_qpbatch<T, R, block, cell> (kCellWide: as kCellNarrow)
    size_t (*smem)(int rows);      // shared memory for a double stack of `rows` rows
};
const QpKernel* qp_kernels(int* n);
const QpKernel* find_qp(int T, int R);     // null when that shape is not compiled

}  // namespace swb
