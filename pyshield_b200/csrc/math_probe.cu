// The device math of mp_math.cuh and the saturation humidity built on it,
// one call per element, for the tests that measure their errors. Part of the
// probe library, not of the C-ABI.
#include <cuda_runtime.h>

#include <cstring>

#include "mp_physics.cuh"
#include "mp_setup.h"

namespace {

using namespace shield;

enum {
  F_DIV = 0, F_SQRT, F_EXP, F_LOG, F_POW, F_QSW, F_QSW_DT, F_QSI, F_QSI_DT,
  // CUDA's functions and the reference's expressions on them, which the forms above replace
  G_EXP, G_LOG, G_POW, G_QSW, G_QSW_DT, G_QSI, G_QSI_DT, G_EXP_LOG
};

// wqs1 and iqs2 (microphysics_funcs.py:52-145) as the reference writes them
__device__ double wqs_cuda(const MpConst& K, double ta, double den) {
  return (K.E00 * exp((K.DC_VAP * log(ta / K.TICE) + K.LV0 * (ta - K.TICE) / (ta * K.TICE)) / K.RVGAS)) /
         (K.RVGAS * ta * den);
}
__device__ double iqs_cuda(const MpConst& K, double ta, double den, double& dqdt) {
  if (ta < K.TICE) {
    if (ta < K.T_SAT_MIN) ta = K.T_SAT_MIN;
    const double q = (K.E00 * exp((K.D2ICE * log(ta / K.TICE) + K.LI2 * (ta - K.TICE) / (ta * K.TICE)) / K.RVGAS)) /
                     (K.RVGAS * ta * den);
    dqdt = q * (K.D2ICE + K.LI2 / ta) / (K.RVGAS * ta);
    return q;
  }
  if (ta > K.TICE + 102.0) ta = K.TICE + 102.0;
  const double q = wqs_cuda(K, ta, den);
  dqdt = q * (K.DC_VAP + K.LV0 / ta) / (K.RVGAS * ta);
  return q;
}

__global__ void math_kernel(int fn, int n, const double* x, const double* y, double* out,
                            const __grid_constant__ MpConst K) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = y[i];
  double r = 0.0, d = 0.0;
  switch (fn) {
    case F_DIV: r = qdiv(a, b); break;
    case F_SQRT: r = qsqrt(a); break;
    case F_EXP: r = xexp(a); break;
    case F_LOG: r = xlog(a); break;
    case F_POW: r = xpowc(a, b); break;
    case F_QSW: r = wqs1(K, a, b); break;
    case F_QSW_DT: wqs2(K, a, b, d), r = d; break;
    case F_QSI: r = iqs1(K, a, b); break;
    case F_QSI_DT: iqs2(K, a, b, d), r = d; break;
    case G_EXP: r = exp(a); break;
    case G_LOG: r = log(a); break;
    case G_POW: r = pow(a, b); break;
    case G_QSW: r = wqs_cuda(K, a, b); break;
    case G_QSW_DT: r = wqs_cuda(K, a, b) * (K.DC_VAP + K.LV0 / a) / (K.RVGAS * a); break;
    case G_QSI: r = iqs_cuda(K, a, b, d); break;
    case G_QSI_DT: iqs_cuda(K, a, b, d), r = d; break;
    case G_EXP_LOG: r = exp(b * log(a)); break;
  }
  out[i] = r;
}

}  // namespace

// out[i] = function `fn` of (x[i], y[i]) for n elements on `stream`: a / b,
// sqrt, exp, log, x^y, then wqs1, its derivative, iqs1, its derivative at
// temperature x and density y; then CUDA's exp, log and pow, the
// saturation humidities as the reference's expressions of them, and
// exp(y log x).
#ifndef PROBE_MATH
#define PROBE_MATH shield_probe_math
#endif
extern "C" int PROBE_MATH(int fn, int n, const double* x, const double* y, double* out, void* stream) {
  if (fn < F_DIV || fn > G_EXP_LOG || n < 1 || !x || !y || !out) return -1;
  ShieldMpConfig cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  MpConst K;
  std::memset(&K, 0, sizeof(K));
  setupm(cfg, K);
  math_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(fn, n, x, y, out, K);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
