// Mixed-precision form of the microphysics step: process rates in FP32,
// saturation adjustment, sedimentation, precipitation and every state
// update in FP64 (see mp_physics_mixed.cuh). FMA contraction is allowed here.
#include "mp_kernel.cuh"
#include "mp_launch.h"

namespace shield {

cudaError_t mp_launch_mixed(const MpArgs& A, cudaStream_t st) { return launch_shapes<true, false>(A, st); }

// Ensemble launch over nz in (64, 128]; the shapes of
// mp_launch_ensemble_plain.
cudaError_t mp_launch_ensemble_mixed(const MpArgs* members, const int64_t* offs, int nm, int nz, int G, int grid,
                                     unsigned long long* counter, cudaStream_t st) {
  if (nz <= PACK80_LMAX) {
    if (G == 2) return launch_ensemble<PackedLayout<5, 2, 1>, 4, true>(members, offs, nm, counter, grid, st);
    if (G == 4) return launch_ensemble<PackedLayout<5, 2, 2>, 2, true>(members, offs, nm, counter, grid, st);
    if (G == 6) return launch_ensemble<PackedLayout<5, 2, 3>, 1, true>(members, offs, nm, counter, grid, st);
    if (G == 8) return launch_ensemble<PackedLayout<5, 2, 4>, 1, true>(members, offs, nm, counter, grid, st);
  } else if (nz <= 96) {
    if (G == 1) return launch_ensemble<ColumnLayout<3, 1>, 8, true>(members, offs, nm, counter, grid, st);
    if (G == 2) return launch_ensemble<ColumnLayout<3, 2>, 4, true>(members, offs, nm, counter, grid, st);
    if (G == 4) return launch_ensemble<ColumnLayout<3, 4>, 2, true>(members, offs, nm, counter, grid, st);
  } else if (nz <= 128) {
    if (G == 1) return launch_ensemble<ColumnLayout<4, 1>, 6, true>(members, offs, nm, counter, grid, st);
    if (G == 2) return launch_ensemble<ColumnLayout<4, 2>, 3, true>(members, offs, nm, counter, grid, st);
    if (G == 4) return launch_ensemble<ColumnLayout<4, 4>, 1, true>(members, offs, nm, counter, grid, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace shield
