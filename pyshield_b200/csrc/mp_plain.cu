// Plain FP64 form of the microphysics step. Compiled with -fmad=false so
// that every multiply and add rounds as the reference's numpy expressions do;
// exp, log, powers and the saturation humidities are those of mp_math.cuh.
#include "mp_kernel.cuh"
#include "mp_launch.h"

namespace shield {

// de_ice (microphysics.py:110-120): applied in place before the step.
__global__ void de_ice_kernel(const __grid_constant__ MpArgs A, Fld3 qi_dt, Fld3 qs_dt) {
  const MpConst& K = A.K;
  const int64_t n = A.ncol * (int64_t)A.nz;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = e % A.ncol, k = e / A.ncol;
    const int64_t i = c % A.nx, j = c / A.nx;
    double* qi = A.in[IN_QI].p + i * A.in[IN_QI].si + j * A.in[IN_QI].sj + k * A.in[IN_QI].sk;
    double* qs = A.in[IN_QS].p + i * A.in[IN_QS].si + j * A.in[IN_QS].sj + k * A.in[IN_QS].sk;
    double* pqi = qi_dt.p + i * qi_dt.si + j * qi_dt.sj + k * qi_dt.sk;
    double* pqs = qs_dt.p + i * qs_dt.si + j * qs_dt.sj + k * qs_dt.sk;
    const double qio = *qi - K.timestep * *pqi;
    const double qin = fmax(qio, K.qi0_max);
    if (*qi > qin) {
      *qs = *qs + *qi - qin;
      *qi = qin;
      const double dqi = (qin - qio) * K.rdt;
      *pqs = *pqs + *pqi - dqi;
      *pqi = dqi;
    }
  }
}


namespace {

__global__ void gather2d(const double* p, int64_t si, int64_t sj, int nx, int64_t n, double* out) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
    out[c] = p[(c % nx) * si + (c / nx) * sj];
}

}  // namespace

int mp_max_levels() { return 256; }

cudaError_t mp_launch_plain(const MpArgs& A, cudaStream_t st) { return launch_shapes<false, false>(A, st); }

// The same launches with the column flags recorded (A.flags non-null).
cudaError_t mp_launch_plain_flags(const MpArgs& A, cudaStream_t st) { return launch_shapes<false, true>(A, st); }

cudaError_t mp_launch_mixed(const MpArgs& A, cudaStream_t st);

cudaError_t mp_launch_step(const MpArgs& A, int precision, cudaStream_t st) {
  if (precision == 1) return mp_launch_mixed(A, st);
  return mp_launch_plain(A, st);
}

cudaError_t mp_launch_de_ice(const MpArgs& A, Fld3 qi_dt, Fld3 qs_dt, cudaStream_t st) {
  const int64_t n = A.ncol * (int64_t)A.nz;
  const int64_t nb = (n + 255) / 256;
  de_ice_kernel<<<(unsigned)(nb < 148 * 16 ? nb : 148 * 16), 256, 0, st>>>(A, qi_dt, qs_dt);
  return cudaGetLastError();
}

cudaError_t mp_gather_area(const double* p, int64_t si, int64_t sj, int nx, int ny, double* out) {
  const int64_t n = (int64_t)nx * ny;
  const int64_t nb = (n + 255) / 256;
  gather2d<<<(unsigned)(nb < 4096 ? nb : 4096), 256>>>(p, si, sj, nx, n, out);
  return cudaGetLastError();
}


// Ensemble launch over nz in (64, 128]: G columns per block, a persistent
// grid of `grid` blocks. 65..80 levels: G = 2, 4, 6 or 8 (1 to 4 groups of
// two packed columns; 640 threads per SM where the block size allows);
// 81..128 levels: G = 1, 2 or 4.
cudaError_t mp_launch_ensemble_plain(const MpArgs* members, const int64_t* offs, int nm, int nz, int G, int grid,
                                     unsigned long long* counter, cudaStream_t st) {
  if (nz <= PACK80_LMAX) {
    if (G == 2) return launch_ensemble<PackedLayout<5, 2, 1>, 4, false>(members, offs, nm, counter, grid, st);
    if (G == 4) return launch_ensemble<PackedLayout<5, 2, 2>, 2, false>(members, offs, nm, counter, grid, st);
    if (G == 6) return launch_ensemble<PackedLayout<5, 2, 3>, 1, false>(members, offs, nm, counter, grid, st);
    if (G == 8) return launch_ensemble<PackedLayout<5, 2, 4>, 1, false>(members, offs, nm, counter, grid, st);
  } else if (nz <= 96) {
    if (G == 1) return launch_ensemble<ColumnLayout<3, 1>, 8, false>(members, offs, nm, counter, grid, st);
    if (G == 2) return launch_ensemble<ColumnLayout<3, 2>, 4, false>(members, offs, nm, counter, grid, st);
    if (G == 4) return launch_ensemble<ColumnLayout<3, 4>, 2, false>(members, offs, nm, counter, grid, st);
  } else if (nz <= 128) {
    if (G == 1) return launch_ensemble<ColumnLayout<4, 1>, 6, false>(members, offs, nm, counter, grid, st);
    if (G == 2) return launch_ensemble<ColumnLayout<4, 2>, 3, false>(members, offs, nm, counter, grid, st);
    if (G == 4) return launch_ensemble<ColumnLayout<4, 4>, 1, false>(members, offs, nm, counter, grid, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace shield
