// kernels_fp64_one.cu -- the FP64 stage kernels for a single grid (ONE), compiled as
// kernels_fp64.cu is, in a unit of their own.
#include "kernel_table.h"
#include "stage_kernel.cuh"

namespace chimera {

namespace {
template <int TX, int TY, int NT, int MINB, bool TMA>
void fill_one(KernelSet* ks) {
#define CHIMERA_ENTRY(S, K)                                                                                   \
  ks->stage[S - 1][K - 1].one = (const void*)&stage_kernel<double, S, K, TX, TY, NT, MINB, false, TMA, UNIT_FP64, \
                                                           false, false, true>
  CHIMERA_ENTRY(1, 1); CHIMERA_ENTRY(1, 2); CHIMERA_ENTRY(1, 3);
  CHIMERA_ENTRY(2, 1); CHIMERA_ENTRY(2, 2); CHIMERA_ENTRY(2, 3);
  CHIMERA_ENTRY(3, 1); CHIMERA_ENTRY(3, 2); CHIMERA_ENTRY(3, 3);
#undef CHIMERA_ENTRY
}
}  // namespace

// The variants a new single-grid handle may start on, and the TMA tile of batches.
void fp64_one_kernels(int variant, KernelSet* ks) {
  switch (variant) {
    case 0: fill_one<32, 16, 256, 2, true>(ks); break;
    case 7: fill_one<8, 8, 192, 2, false>(ks); break;
    case 8: fill_one<16, 8, 192, 2, false>(ks); break;
    case 9: fill_one<16, 16, 320, 2, false>(ks); break;
    case 10: fill_one<32, 15, 384, 2, true>(ks); break;
    case 11: fill_one<64, 16, 768, 1, true>(ks); break;
    default: break;
  }
}

}  // namespace chimera
