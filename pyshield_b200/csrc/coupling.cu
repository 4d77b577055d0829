// Physics-to-dynamics column coupling kernels (compiled with -fmad=false).
//
//  * update_physics_state_with_tendencies  pySHiELD/stencils/physics.py:146-194
//  * fill_gfs_delp                         pySHiELD/update/update_atmos_state.py:21-37
//  * prepare_tendencies_and_update_tracers pySHiELD/update/update_atmos_state.py:40-92
//  * moist_cv                              pySHiELD/update/fv_update_phys.py:20-51
//  * update_pressure_and_surface_winds     pySHiELD/update/fv_update_phys.py:54-75
//  * copy_dycore_to_physics                pySHiELD/update/update_atmos_state.py:95-142
//
// All are HBM-streaming work. The first is elementwise (one thread per point,
// the fastest-varying storage dimension mapped to consecutive threads), as
// is the dycore-to-physics copy. The other four are fused into one kernel
// over tiles of columns that runs them in the reference's order, so that the
// updated vapour, delp, pt and tendencies pass from one stencil to the next
// in registers and shared memory instead of HBM.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/shield_mp.h"

namespace shield {
void set_last_error(const std::string& msg);
}

namespace {

struct F3 {
  double* p;
  int64_t si, sj, sk;
  __device__ __forceinline__ double& at(int64_t i, int64_t j, int64_t k) const { return p[i * si + j * sj + k * sk]; }
};

F3 mk(const ShieldField3D& f) { return F3{f.ptr, f.si, f.sj, f.sk}; }

struct UpdArgs {
  F3 x[10], t[10], o[10];
  int nx, ny, nz;
  int kfast;
  double dt;
};

// The two field kernels below work per field and per stretch of lines: a
// block handles one field (blockIdx.z) over LINES consecutive lines of the
// domain, a line being a (j, k) row (or, with k fastest in memory, an (i, j)
// column) whose points lie on consecutive threads. Its reads, then its
// writes, are contiguous stretches of a few storages instead of short lines
// of many, which keeps DRAM pages open. All of a block's loads are issued
// before its stores; index arithmetic is 32-bit (the entry points check the
// box).
constexpr int LINES = 8;
__device__ __forceinline__ void line_ijk(int kfast, int nx, int ny, int row, int t, int& i, int& j, int& k) {
  if (kfast) {
    k = t;
    i = row % nx;
    j = row / nx;
  } else {
    i = t;
    j = row % ny;
    k = row / ny;
  }
}

__global__ void update_physics_state_kernel(const __grid_constant__ UpdArgs A) {
  const int rows = A.kfast ? A.nx * A.ny : A.ny * A.nz;
  const int len = A.kfast ? A.nz : A.nx;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= len) return;
  const F3& X = A.x[blockIdx.z];
  const F3& T = A.t[blockIdx.z];
  const F3& O = A.o[blockIdx.z];
  for (int r0 = blockIdx.y * LINES; r0 < rows; r0 += gridDim.y * LINES) {
    double x[LINES], d[LINES];
    int64_t oo[LINES];
#pragma unroll
    for (int b = 0; b < LINES; ++b) {
      int i, j, k;
      line_ijk(A.kfast, A.nx, A.ny, r0 + b < rows ? r0 + b : rows - 1, t, i, j, k);
      x[b] = X.at(i, j, k);
      d[b] = T.at(i, j, k);
      oo[b] = i * O.si + j * O.sj + k * O.sk;
    }
#pragma unroll
    for (int b = 0; b < LINES; ++b)
      if (r0 + b < rows) O.p[oo[b]] = x[b] + d[b] * A.dt;
  }
}

enum {
  U_DT = 0, V_DT, PT_DT, U_T1, V_T1, PU_PT, PU_QV, PU_QL, PU_QR, PU_QS, PU_QI, PU_QG, U_T0, V_T0, PT_T0,
  D_QV, D_QL, D_QR, D_QS, D_QI, D_QG, PRSI, D_DELP, D_PT, PE, PELN, PK, D_UA, D_VA, N_ATM
};

struct AtmArgs {
  F3 f[N_ATM];
  F3 ps, us, vs;
  int nx, ny, nz, hx, mode;
  double rdt, dt, kappa, cp_air;
  double CV_AIR, CV_VAP, C_LIQ, C_ICE;
};

// The column stencils of UpdateAtmosphereState in one kernel. A block owns
// AT_TC = 32 consecutive columns of the full domain (lane = column: every
// level's accesses are coalesced in the i-fastest layout) and has AT_LW warps
// share their levels. The pointwise work runs level-parallel; the
// level-by-level recurrences run in one warp over shared-memory columns, in
// the reference's order:
//   1 (all warps)  the vapour and delp of every level into shared memory;
//   2 (one warp)   fill_gfs_delp's three sweeps, where some column of the
//                  block has a level they change;
//   3 (all warps)  the filled vapour back (full domain); on the compute
//                  domain prepare_tendencies_and_update_tracers and moist_cv
//                  level by level (moist_cv reads what prepare wrote at the
//                  same level); the new delp into shared memory;
//   4 (one warp)   update_pressure_and_surface_winds' pe sum;
//   5 (all warps)  pe, peln, pk.
// SAME: every field has one set of strides (NDSL storages of one shape), so
// a level has one offset instead of 29.
//
// Bound by memory latency and short rows (256 B of a field and level at a
// time): 1.39 GB at C96 L79, 0.212 ms at the measured copy rate. Shapes
// (columns x level warps, blocks per SM; ms at C96 L79 / C96 L127 / 37 x 41
// L79): 32 x 4, 3 blocks, a general offset per field 0.397 / 0.755 / 0.066;
// one offset and 32 x 4, 4 blocks 0.388 / 0.704 / 0.070; 32 x 8, 4 blocks
// 0.347 / 0.578 / 0.049; 32 x 16, 2 blocks 0.327 / 0.546 / 0.039; 64 x 8,
// 2 blocks 0.324 / 0.642 / 0.054; 128 x 8, one block 0.370. More warps give
// each phase more loads in flight; beyond 32 a SM the registers spill (48
// warps 0.406). Without phases 4 and 5 the launch takes 0.288.
// Phase 2 by need (C96 L79 / L127): 0.286 / 0.437 where no level of any column
// needs it, 0.329 / 0.546 with needy halo columns alone (a third of the blocks),
// 0.326 / 0.499 with 1 % of the levels needy and 0.335 / 0.507 with every other
// one, both sweeps in every block; always swept, with an offset per field and
// 4 level warps, 0.384 to 0.400 / 0.730 to 0.751.
constexpr int AT_TC = 32, AT_LW = 16, AT_MINB = 2;

template <bool SAME>
__global__ void __launch_bounds__(AT_TC * AT_LW, AT_MINB) update_atmos_state_kernel(const __grid_constant__ AtmArgs A) {
  // rows of AT_TC columns: the vapour fill_gfs_delp works on, then the dycore
  // delp it reads; later prepare's new delp (each level's thread replaces
  // its own), then the interface pressure
  extern __shared__ double smem[];
  const int nk = A.nz + 1;  // the reference builds these stencils on nz + 1 levels
  const int cx = threadIdx.x % AT_TC, w = threadIdx.x / AT_TC;
  double* const sq = smem + cx;
  double* const sd = smem + (size_t)nk * AT_TC + cx;
  const int nxf = A.nx + 2 * A.hx;
  const int ncf = nxf * (A.ny + 2 * A.hx);
  const int c = blockIdx.x * AT_TC + cx;
  const bool live = c < ncf;
  const int i = live ? c % nxf - A.hx : 0, j = live ? c / nxf - A.hx : 0;
  const bool compute = live && i >= 0 && j >= 0 && i < A.nx && j < A.ny;
  const bool dycore_only = (A.mode & SHIELD_UAS_DYCORE_ONLY) != 0;
  const bool apply = (A.mode & SHIELD_UAS_APPLY) != 0;
  const F3* f = A.f;
  const int64_t o0 = i * f[0].si + j * f[0].sj, ok = f[0].sk;
  auto at = [&](const F3& F, int k) -> double& { return SAME ? F.p[o0 + k * ok] : F.at(i, j, k); };
  const F3& Q = dycore_only ? f[D_QV] : f[PU_QV];
  const F3& DP = f[D_DELP];
  const double q_min = 1.0e-9;

  // ---- 1: fill_gfs_delp's inputs, levels 0 .. nk - 2
  bool fill = false;  // a level that the sweeps would change
  if (live) {
#pragma unroll 4
    for (int k = w; k < nk - 1; k += AT_LW) {
      const double q = at(Q, k), dp = at(DP, k);
      sq[k * AT_TC] = q;
      sd[k * AT_TC] = dp;
      fill = fill || (k > 0 ? q < q_min : q < 0.0);
    }
  }
  // ---- 2: fill_gfs_delp(delp, q, 1e-9) (update_atmos_state.py:21-37)
  if (__syncthreads_or(fill)) {
    if (w == 0 && live) {
      // BACKWARD interval(0, -2): borrow from the (updated) level below
      double qn = sq[(nk - 2) * AT_TC];
      double dpn = sd[(nk - 2) * AT_TC];
      for (int k = nk - 3; k >= 0; --k) {
        double qk = sq[k * AT_TC];
        const double dpk = sd[k * AT_TC];
        if (qn < q_min) qk = qk + (qn - q_min) * dpn / dpk;
        sq[k * AT_TC] = qk;
        qn = qk;
        dpn = dpk;
      }
      // PARALLEL interval(1, -1) clamp, FORWARD interval(1, -1) borrow, FORWARD
      // interval(0, -1) zero: the borrow chain runs on the unzeroed values
      double qprev = sq[0];
      double dprev = sd[0];
      if (qprev < 0.0) sq[0] = 0.0;
      for (int k = 1; k < nk - 1; ++k) {
        double qk = sq[k * AT_TC];
        const double dpk = sd[k * AT_TC];
        if (qk < q_min) qk = q_min;
        if (qprev < 0.0) qk = qk + qprev * (dprev) / (dpk);
        qprev = qk;
        dprev = dpk;
        sq[k * AT_TC] = (qk < 0.0) ? 0.0 : qk;
      }
    }
    __syncthreads();
  }
  // ---- 3: the filled vapour; prepare_tendencies_and_update_tracers and moist_cv.
  // Every load of a level comes before its first store: the fields are
  // separate storages, but the compiler cannot know that, and a store
  // between two loads would make each group of loads wait for the last.
  for (int k = w; k < nk; k += AT_LW) {
    const bool filled = live && k < nk - 1;
    if (dycore_only || !compute) {
      if (filled) at(Q, k) = sq[k * AT_TC];
      continue;
    }
    const bool prep = k < nk - 1;
    // loads
    double dq[6];
    dq[0] = at(f[D_QV], k);
    dq[1] = at(f[D_QL], k);
    dq[2] = at(f[D_QR], k);
    dq[3] = at(f[D_QS], k);
    dq[4] = at(f[D_QI], k);
    dq[5] = at(f[D_QG], k);
    double pt_dt = at(f[PT_DT], k);
    const double pt = apply ? at(f[D_PT], k) : 0.0;
    double u_dt = 0.0, v_dt = 0.0, pq[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, dp = 0.0;
    if (prep) {
      u_dt = at(f[U_DT], k) + (at(f[U_T1], k) - at(f[U_T0], k)) * A.rdt;
      v_dt = at(f[V_DT], k) + (at(f[V_T1], k) - at(f[V_T0], k)) * A.rdt;
      pt_dt = pt_dt + (at(f[PU_PT], k) - at(f[PT_T0], k)) * A.rdt;
      dp = at(f[PRSI], k + 1) - at(f[PRSI], k);
      pq[0] = sq[k * AT_TC];
      pq[1] = at(f[PU_QL], k);
      pq[2] = at(f[PU_QR], k);
      pq[3] = at(f[PU_QS], k);
      pq[4] = at(f[PU_QI], k);
      pq[5] = at(f[PU_QG], k);
    }
    // prepare_tendencies_and_update_tracers, interval(0, -1)
    double q0 = 0.0;
    if (prep) {
      double qw[6];
      for (int t = 0; t < 6; ++t) qw[t] = dp * pq[t];
      const double qt = qw[0] + qw[1] + qw[2] + qw[3] + qw[4] + qw[5];
      const double q_sum = dq[0] + dq[1] + dq[2] + dq[3] + dq[4] + dq[5];
      q0 = sd[k * AT_TC] * (1.0 - q_sum) + qt;  // the old delp, read before the store below
      for (int t = 0; t < 6; ++t) dq[t] = qw[t] / q0;
    }
    // moist_cv(dycore q..., dycore pt, t_dt = pt_dt, CP_AIR, dt), nz + 1 levels
    double pt_new = 0.0;
    if (apply) {
      const double ql = dq[1] + dq[2];
      const double qs = dq[4] + dq[3] + dq[5];
      const double gz = ql + qs;
      const double qv = dq[0];
      const double cvm = (1.0 - (qv + gz)) * A.CV_AIR + qv * A.CV_VAP + ql * A.C_LIQ + qs * A.C_ICE;
      pt_new = pt + pt_dt * A.dt * A.cp_air / cvm;
    }
    // stores
    if (filled) at(Q, k) = sq[k * AT_TC];
    if (prep) {
      at(f[U_DT], k) = u_dt;
      at(f[V_DT], k) = v_dt;
      at(f[D_DELP], k) = q0;
      sd[k * AT_TC] = q0;
      at(f[D_QV], k) = dq[0];
      at(f[D_QL], k) = dq[1];
      at(f[D_QR], k) = dq[2];
      at(f[D_QS], k) = dq[3];
      at(f[D_QI], k) = dq[4];
      at(f[D_QG], k) = dq[5];
    }
    if (apply) {
      at(f[D_PT], k) = pt_new;
      at(f[PT_DT], k) = 0.0;
    } else if (prep) {
      at(f[PT_DT], k) = pt_dt;
    }
  }
  if (dycore_only || !apply) return;  // block-uniform: the mode is the launch's
  __syncthreads();
  // ---- 4: update_pressure_and_surface_winds' sum, pe[k] = pe[k - 1] + delp[k - 1]
  if (w == 0 && compute) {
    double pe = at(f[PE], 0);
    double dprev = sd[0];
#pragma unroll 8
    for (int k = 1; k < nk; ++k) {
      pe = pe + dprev;
      dprev = k < nk - 1 ? sd[k * AT_TC] : 0.0;
      sd[k * AT_TC] = pe;
    }
  }
  __syncthreads();
  // ---- 5: pe, peln, pk on levels 1 .. nk - 1; ps and the surface winds
  for (int k = 1 + w; k < nk; k += AT_LW) {
    if (!compute) continue;
    const double pe = sd[k * AT_TC];
    at(f[PE], k) = pe;
    const double peln = log(pe);
    at(f[PELN], k) = peln;
    at(f[PK], k) = exp(A.kappa * peln);
  }
  if (w == 0 && compute) {
    A.ps.at(i, j, 0) = sd[(nk - 1) * AT_TC];
    A.us.at(i, j, 0) = at(f[D_UA], nk - 2);
    A.vs.at(i, j, 0) = at(f[D_VA], nk - 2);
  }
}

cudaError_t launch_atmos(const AtmArgs& A, int ncf, cudaStream_t st) {
  bool same = true;
  for (const F3& F : A.f) same = same && F.si == A.f[0].si && F.sj == A.f[0].sj && F.sk == A.f[0].sk;
  auto kern = same ? update_atmos_state_kernel<true> : update_atmos_state_kernel<false>;
  const size_t smem = sizeof(double) * 2 * AT_TC * (size_t)(A.nz + 1);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)((ncf + AT_TC - 1) / AT_TC), AT_TC * AT_LW, smem, st>>>(A);
  return cudaGetLastError();
}

// DycoreToPhysics' copy of 16 fields (update_atmos_state.py:95-142, built at
// :160-167 on the compute domain plus one interface point in x and y,
// PARALLEL interval(0, -1) of nz + 1 levels), the fastest-varying storage
// dimension on consecutive threads.
constexpr int N_D2P = 16;
struct D2PArgs {
  F3 in[N_D2P], out[N_D2P];
  int nx1, ny1, nz;  // the box: nx + 1, ny + 1, nz
  int kfast;
};

// The copy, per field and stretch of lines as update_physics_state_kernel.
__global__ void copy_dycore_to_physics_kernel(const __grid_constant__ D2PArgs A) {
  const int rows = A.kfast ? A.nx1 * A.ny1 : A.ny1 * A.nz;
  const int len = A.kfast ? A.nz : A.nx1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= len) return;
  const F3& src = A.in[blockIdx.z];
  const F3& dst = A.out[blockIdx.z];
  for (int r0 = blockIdx.y * LINES; r0 < rows; r0 += gridDim.y * LINES) {
    double v[LINES];
    int64_t od[LINES];
#pragma unroll
    for (int b = 0; b < LINES; ++b) {
      int i, j, k;
      line_ijk(A.kfast, A.nx1, A.ny1, r0 + b < rows ? r0 + b : rows - 1, t, i, j, k);
      v[b] = src.at(i, j, k);
      od[b] = i * dst.si + j * dst.sj + k * dst.sk;
    }
#pragma unroll
    for (int b = 0; b < LINES; ++b)
      if (r0 + b < rows) dst.p[od[b]] = v[b];
  }
}

// 2-D launch over (line length, rows): 128 threads along a line, at most
// 65,535 block rows (a grid-stride loop covers the rest)
dim3 line_grid(int64_t len, int64_t rows) {
  const int64_t bx = (len + 127) / 128;
  return dim3((unsigned)bx, (unsigned)(rows < 65535 ? (rows > 0 ? rows : 1) : 65535));
}

}  // namespace

extern "C" int shield_update_physics_state(int nx, int ny, int nz, const ShieldField3D* state10,
                                           const ShieldField3D* tend10, const ShieldField3D* out10, double dt,
                                           void* stream) {
  if (!state10 || !tend10 || !out10 || nx < 1 || ny < 1 || nz < 1) {
    shield::set_last_error("shield_update_physics_state: bad arguments");
    return SHIELD_EINVAL;
  }
  UpdArgs A;
  for (int p = 0; p < 10; ++p) {
    if (!state10[p].ptr || !tend10[p].ptr || !out10[p].ptr) {
      shield::set_last_error("shield_update_physics_state: null field");
      return SHIELD_EINVAL;
    }
    A.x[p] = mk(state10[p]);
    A.t[p] = mk(tend10[p]);
    A.o[p] = mk(out10[p]);
  }
  A.nx = nx;
  A.ny = ny;
  A.nz = nz;
  A.kfast = (state10[0].sk == 1) ? 1 : 0;
  A.dt = dt;
  const int64_t len = A.kfast ? nz : nx, rows = A.kfast ? (int64_t)nx * ny : (int64_t)ny * nz;
  if (rows * len > INT32_MAX) {
    shield::set_last_error("shield_update_physics_state: box too large for 32-bit indices");
    return SHIELD_ELAYOUT;
  }
  dim3 grid = line_grid(len, (rows + LINES - 1) / LINES);
  grid.z = 10;
  update_physics_state_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(A);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    shield::set_last_error(std::string("shield_update_physics_state: ") + cudaGetErrorString(e));
    return SHIELD_ECUDA;
  }
  return SHIELD_OK;
}

extern "C" int shield_update_atmos_state(int nx, int ny, int nz, int hx, int mode, const ShieldField3D* f, ShieldField3D ps,
                                         ShieldField3D u_srf, ShieldField3D v_srf, double rdt, double dt, double kappa,
                                         double cp_air, void* stream) {
  if (!f || nx < 1 || ny < 1 || nz < 2 || hx < 0 || !ps.ptr || !u_srf.ptr || !v_srf.ptr) {
    shield::set_last_error("shield_update_atmos_state: bad arguments");
    return SHIELD_EINVAL;
  }
  if (nz > 128) {
    shield::set_last_error("shield_update_atmos_state: nz > 128 is not supported");
    return SHIELD_ELAYOUT;
  }
  AtmArgs A;
  for (int p = 0; p < N_ATM; ++p) {
    if (!f[p].ptr) {
      shield::set_last_error("shield_update_atmos_state: null field " + std::to_string(p));
      return SHIELD_EINVAL;
    }
    A.f[p] = mk(f[p]);
  }
  A.ps = mk(ps);
  A.us = mk(u_srf);
  A.vs = mk(v_srf);
  A.nx = nx;
  A.ny = ny;
  A.nz = nz;
  A.hx = hx;
  A.mode = mode;
  A.rdt = rdt;
  A.dt = dt;
  A.kappa = kappa;
  A.cp_air = cp_air;
  // the constants of pyshield_b200/constants.py
  const double RVGAS = 461.50, RDGAS = 287.05, CP_AIR = 1004.6;
  A.CV_AIR = CP_AIR - RDGAS;
  A.CV_VAP = 3.0 * RVGAS;
  A.C_LIQ = 4.1855e3;
  A.C_ICE = 1972.0;
  const int64_t ncf = (int64_t)(nx + 2 * hx) * (ny + 2 * hx);
  if (ncf > INT32_MAX) {
    shield::set_last_error("shield_update_atmos_state: more than 2^31 - 1 columns");
    return SHIELD_ELAYOUT;
  }
  cudaError_t e = launch_atmos(A, (int)ncf, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    shield::set_last_error(std::string("shield_update_atmos_state: ") + cudaGetErrorString(e));
    return SHIELD_ECUDA;
  }
  return SHIELD_OK;
}

extern "C" int shield_copy_dycore_to_physics(int nx, int ny, int nz, const ShieldField3D* dycore16,
                                             const ShieldField3D* physics16, void* stream) {
  if (!dycore16 || !physics16 || nx < 1 || ny < 1 || nz < 1) {
    shield::set_last_error("shield_copy_dycore_to_physics: bad arguments");
    return SHIELD_EINVAL;
  }
  D2PArgs A;
  for (int p = 0; p < N_D2P; ++p) {
    if (!dycore16[p].ptr || !physics16[p].ptr) {
      shield::set_last_error("shield_copy_dycore_to_physics: null field " + std::to_string(p));
      return SHIELD_EINVAL;
    }
    A.in[p] = mk(dycore16[p]);
    A.out[p] = mk(physics16[p]);
  }
  A.nx1 = nx + 1;
  A.ny1 = ny + 1;
  A.nz = nz;
  A.kfast = (physics16[0].sk == 1) ? 1 : 0;
  const int64_t len = A.kfast ? nz : A.nx1, rows = A.kfast ? (int64_t)A.nx1 * A.ny1 : (int64_t)A.ny1 * nz;
  if (rows * len > INT32_MAX) {
    shield::set_last_error("shield_copy_dycore_to_physics: box too large for 32-bit indices");
    return SHIELD_ELAYOUT;
  }
  dim3 grid = line_grid(len, (rows + LINES - 1) / LINES);
  grid.z = N_D2P;
  copy_dycore_to_physics_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(A);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    shield::set_last_error(std::string("shield_copy_dycore_to_physics: ") + cudaGetErrorString(e));
    return SHIELD_ECUDA;
  }
  return SHIELD_OK;
}
