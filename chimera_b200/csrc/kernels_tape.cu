// kernels_tape.cu -- the adjoint's forward re-run: the FP64 stage kernels with
// the tape (TapeOut).  Compiled with --fmad=false like the plain FP64 form, whose
// bits they reproduce.
#include "kernel_table.h"
#include "stage_kernel.cuh"

namespace chimera {

namespace {
template <int TX, int TY, int NT, int MINB, bool MIXBC = false>
void fill(KernelSet* ks) {
  const size_t smem = TileGeom<TX, TY>::template smem_bytes<double>();
#define CHIMERA_ENTRY(S, K) \
  ks->stage[S - 1][K - 1] = KernelEntry{                                                                  \
      (const void*)&stage_kernel<double, S, K, TX, TY, NT, MINB, false, false, UNIT_TAPE, MIXBC, true, true>, \
                                        smem, TX, TY, NT}
  CHIMERA_ENTRY(1, 1); CHIMERA_ENTRY(1, 2); CHIMERA_ENTRY(1, 3);
  CHIMERA_ENTRY(2, 1); CHIMERA_ENTRY(2, 2); CHIMERA_ENTRY(2, 3);
  CHIMERA_ENTRY(3, 1); CHIMERA_ENTRY(3, 2); CHIMERA_ENTRY(3, 3);
#undef CHIMERA_ENTRY
  ks->cfl = KernelEntry{};
  ks->elem_bytes = 8;
}
}  // namespace

// small: 8 x 8 tiles, for grids of which the device holds all of them at once
void tape_kernels(bool small, KernelSet* out) { small ? fill<8, 8, 192, 2>(out) : fill<32, 15, 384, 2>(out); }
void tape_mixed_pair_kernels(KernelSet* out) { fill<32, 16, 256, 2, true>(out); }

}  // namespace chimera
