// Kernel parameter block of the microphysics step (host and device).
#pragma once

#include <cstdint>

// The device code of a unit that keeps IEEE rounding (SHIELD_IEEE, see
// mp_math.cuh) lives in a namespace of its own.
#ifdef SHIELD_IEEE
#define SHIELD_ARITH ieee
#else
#define SHIELD_ARITH quick
#endif

namespace shield {

// The physical constants (pyshield_b200/constants.py), for the functions that
// want them as literals; setupm copies them into MpConst.
constexpr double PH_RVGAS = 461.50, PH_C_ICE = 1972.0, PH_C_LIQ = 4.1855e3, PH_TICE = 273.16, PH_E00 = 611.21;
constexpr double PH_HLV = 2.5e6, PH_HLF = 3.3358e5, PH_CP_AIR = 1004.6;
constexpr double PH_DC_VAP = 4.0 * PH_RVGAS - PH_C_LIQ, PH_DC_ICE = PH_C_LIQ - PH_C_ICE;
constexpr double PH_D2ICE = PH_DC_VAP + PH_DC_ICE;
constexpr double PH_LV0 = PH_HLV - PH_DC_VAP * PH_TICE, PH_LI00 = PH_HLF - PH_DC_ICE * PH_TICE;
constexpr double PH_LI2 = PH_LV0 + PH_LI00;

// Every scalar the step reads: the physical constants, the process constants
// of Microphysics.setupm (pySHiELD/stencils/microphysics.py:1813-1953), the
// sub-step scalars of _set_timestep (:1964-1979) and the namelist values the
// stencils bake in as externals (:1715-1804).
struct MpConst {
  // physical constants (pyshield_b200/constants.py order)
  double GRAV, RGRAV, RDGAS, RVGAS, HLV, HLF, CP_AIR, KAPPA, CP_VAP, CV_AIR, CV_VAP, C_ICE, C_LIQ, TICE, E00,
      DC_VAP, DC_ICE, D2ICE, LV0, LI00, LI2, EPS, ZVIR, T_MIN, T_SAT_MIN, LAT2;
  // Microphysics.__init__ scalars (:1643-1658, :1712-1713) and init (:1806-1811)
  double c_air, c_vap, d0_vap, lv00, cpaut, so3, zs, log_10, tice0, t_wfr;
  // setupm
  double fac_rc, cracs, csacr, cgacr, cgacs, acco[3][4], csacw, csaci, cgacw, cgaci, cracw, cssub[5], crevp[5],
      cgfr[2], csmlt[5], cgmlt[5], ces0;
  double iqs_lo_num;  // E00 * exp(...) of iqs1's below-T_SAT_MIN branch
  // _set_timestep
  double timestep, rdt, dts, dt_rain, rdts, dt_evap, fac_i2s, fac_g2v, fac_v2g, fac_imlt, fac_l2v;
  int ntimes;
  // namelist values
  double tice, ql_mlt, qs_mlt, t_sub, qi_gen, qi_lim, qi0_max, dw_ocean, dw_land, qc_crt, qi0_crt, qs0_crt, rh_inc,
      rh_inr, vi_fac, vs_fac, vg_fac, vr_fac, vi_max, vs_max, vg_max, vr_max, ccn_l, ccn_o;
  int do_qa, const_vg, const_vi, const_vr, const_vs, rad_snow, rad_rain, do_sedi_heat, do_sedi_w, fast_sat_adj,
      fix_negative, irain_f, prog_ccn, use_ccn, sedi_transport, z_slope_ice, z_slope_liq, de_ice;
  double r_log_10;  // 1 / log_10
};

// FP32 copies of the constants the mixed form's process rates use.
struct MpConstF {
  double qs_rtw;  // 1 / (tice - t_wfr) of the saturation adjustment
  float E00, DC_VAP, LV0, D2ICE, LI2, RVGAS, TICE, T_SAT_MIN, iqs_lo_num, LAT2;
  float cracs, csacr, cgacr, cgacs, acco[3][4], csacw, csaci, cgacw, cgaci, cracw, cssub[5], crevp[5], cgfr[2],
      csmlt[5], cgmlt[5], ces0, log_10, fac_rc, so3, dt_rain, dts, rdts, fac_i2s;
};

// A strided 3-D field; ptr addresses the compute-domain origin.
struct Fld3 {
  double* p;
  int64_t si, sj, sk;
};
struct Fld2 {
  const double* p;
  int64_t si, sj;
};

// n / d for 0 <= n < 2^31 as a multiply and a shift: with 2^(s - 1) < d <= 2^s
// and m = ceil(2^(31 + s) / d), the excess n (m d - 2^(31 + s)) stays below
// 2^(31 + s). (A 64-bit division is about a hundred instructions.)
struct FastDiv {
  uint32_t m, s;
};
inline FastDiv fast_div(int d) {
  FastDiv f{0, 31};
  while ((int64_t(1) << (f.s - 31)) < d) ++f.s;
  f.m = (uint32_t)(((uint64_t(1) << f.s) + (uint64_t)d - 1) / (uint64_t)d);
  return f;
}

// Input tiles staged in shared memory, in this order.
enum InField {
  IN_PT = 0, IN_QV, IN_QL, IN_QR, IN_QI, IN_QS, IN_QG, IN_QA, IN_UA, IN_VA, IN_DELP, IN_DELZ, IN_W, IN_QAZ,
  N_IN
};
// Output slots (tendency increments, then assigned fields), same tiles reused.
enum OutField {
  OUT_PT_DT = 0, OUT_QV_DT, OUT_QL_DT, OUT_QR_DT, OUT_QI_DT, OUT_QS_DT, OUT_QG_DT, OUT_QA_DT, OUT_UDT, OUT_VDT,
  OUT_W, OUT_QAZ, N_OUT
};

struct MpArgs {
  MpConst K;
  MpConstF KF;
  int nx, ny, nz;
  int64_t ncol;
  FastDiv by_nx;
  // the caller's fields all have in[0]'s strides, which are not k-fastest:
  // one offset serves them (set by plan_layout)
  int same_strides;
  Fld3 in[N_IN];
  Fld3 out[N_OUT];
  int fresh;  // the tendencies count as zero on entry: written whole, not added to
  Fld2 land, area;
  double *rain, *snow, *ice, *graupel;  // (ncol,) surface precipitation [mm/day]; may be null
  int* err;                             // device error word
  // column flags of each sub-step (ntimes x ncol, see MpFlagBits), written
  // only by the flag-recording launch; null otherwise
  int* flags;
};

// The staging's precomputed values, from the domain and the fields' strides.
inline void plan_layout(MpArgs& A) {
  A.by_nx = fast_div(A.nx);
  const Fld3& a = A.in[0];
  bool same = a.sk != 1;
  auto like = [&](const Fld3& f) { return f.si == a.si && f.sj == a.sj && f.sk == a.sk; };
  for (int f = 1; f < IN_QAZ; ++f) same = same && like(A.in[f]);
  for (int o = 0; o < OUT_QAZ; ++o) same = same && like(A.out[o]);
  A.same_strides = same ? 1 : 0;
}

// Bits of the per-column, per-sub-step flags word: which species fall (the
// reference's column-wide no_fall == 0, microphysics.py:349-368 for rain in
// each warm_rain pass, :773-1168 for ice, snow and graupel; ice also needs
// vi_fac >= 1e-5) and the melting level, the first level whose stop_k is 1
// (:706-724; the bottom level when no level is warmer than tice).
enum MpFlagBits : unsigned {
  FLAG_RAIN_FALLS_1 = 1u << 0,
  FLAG_RAIN_FALLS_2 = 1u << 1,
  FLAG_ICE_FALLS = 1u << 2,
  FLAG_SNOW_FALLS = 1u << 3,
  FLAG_GRAUPEL_FALLS = 1u << 4,
  FLAG_MELT_SHIFT = 16u,  // melting level in bits 16..23
};

// Parameter block of the adjoint (vector-Jacobian product) launch. in: the
// step's input state (the first 13 input fields, in the order of InField);
// cot: cotangents of the outputs in the order of OutField (the 10
// tendencies, wmp, the cloud-fraction accumulator); grad: the input
// adjoints written by the launch, in the order of InField (the 13 state
// fields, then the accumulator). A null field pointer is a zero cotangent or
// a gradient that is not written. rain_b .. graupel_b: cotangents of the
// surface totals, ncol each, or null.
constexpr int N_VJP_IN = 13;
constexpr int N_VJP_COT = 12;
constexpr int N_VJP_GRAD = 14;
struct VjpArgs {
  MpConst K;
  MpConstF KF;
  int nx, ny, nz;
  int64_t ncol;
  Fld3 in[N_VJP_IN];
  Fld3 cot[N_VJP_COT];
  Fld3 grad[N_VJP_GRAD];
  Fld2 land, area;
  const double *rain_b, *snow_b, *ice_b, *graupel_b;
  // workspace of mp_vjp_workspace_doubles(ntimes, nz * ncol, ncol) doubles
  double* ws;
  // the incoming qi_dt that de_ice reads (null: zero)
  Fld3 de_ice_qi_dt;
};

}  // namespace shield
