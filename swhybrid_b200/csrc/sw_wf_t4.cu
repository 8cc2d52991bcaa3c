// First-pass kernel instantiations for groups of 4 threads per record pair.
#include "sw_wavefront.cuh"
#include "sw_registry.h"

namespace swb {
namespace {
template <int R, int B, int NB = B>
constexpr WfKernel inst() {
    return WfKernel{4, R, B, NB,
                    {(const void*)&sw_wavefront<4, R, B, CellWide>,
                     (const void*)&sw_wavefront<4, R, NB, CellNarrow<0, 0>>,
                     (const void*)&sw_wavefront<4, R, NB, CellNarrow<12, 2>>,
                     (const void*)&sw_wavefront<4, R, NB, CellNarrow<12, 1>>},
                    &wf_smem_bytes<4, R>, (const void*)&sw_batch<4, R, B>};
}
}  // namespace

// rows per thread R (any even number; the two half-columns hold R/2 rows
// each) and the block size that leaves every shape register room with next
// to no spilling (16 rows: up to 16 bytes, 8 stacked: 6, 48 with run-time gap costs:
// 8; block sizes are multiples of 128 threads); 48 rows run 12 warps
// per SM with CellNarrow (6.05 against 5.65 TCUPS at 8) and 8 with CellWide
extern const WfKernel wf_table_t4[] = {
    inst<4, 768>(),  inst<6, 768>(),  inst<8, 768>(),  inst<10, 640>(), inst<12, 640>(),
    inst<16, 640>(), inst<20, 512>(), inst<24, 512>(), inst<28, 384>(), inst<32, 384>(),
    inst<40, 384>(), inst<48, 256, 384>(), inst<56, 256>(), inst<64, 256>(),
};
extern const int wf_table_t4_n = sizeof(wf_table_t4) / sizeof(wf_table_t4[0]);

}  // namespace swb
