// Instantiations of the paired-query batched kernel (sw_qpair.cuh).
#include "sw_qpair.cuh"
#include "sw_registry.h"

namespace swb {
namespace {
template <int T, int R, int B>
constexpr QpKernel qinst() {
    return QpKernel{T, R, B,
                    {(const void*)&sw_qpbatch<T, R, B, CellNarrow<0, 0>>,
                     (const void*)&sw_qpbatch<T, R, B, CellNarrow<0, 0>>,
                     (const void*)&sw_qpbatch<T, R, B, CellNarrow<12, 2>>,
                     (const void*)&sw_qpbatch<T, R, B, CellNarrow<12, 1>>},
                    &qp_smem_bytes<T, R>};
}
}  // namespace

// Block sizes as for the same shapes of the other first-pass kernels; none of
// them spills (157..253 registers).  ms for 64 queries of 50..5,000 residues
// against 57,000 records, gap costs 10/2 and 8/2 (at run time): 16x64 227 and
// 230, 16x48 229 and 237, 16x32 219 and 223, 32x32 223 and 239, 8x64 225 and 237.
extern const QpKernel qp_table[] = {
    qinst<16, 64, 256>(), qinst<16, 48, 256>(), qinst<16, 32, 384>(), qinst<32, 32, 384>(),
    qinst<8, 64, 256>(),
};
extern const int qp_table_n = sizeof(qp_table) / sizeof(qp_table[0]);

const QpKernel* qp_kernels(int* n) {
    *n = qp_table_n;
    return qp_table;
}

}  // namespace swb
