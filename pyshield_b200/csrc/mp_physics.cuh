// Pointwise GFDL microphysics processes for one model level, on the device.
//
// Each function restates one function of pySHiELD's
// pySHiELD/functions/microphysics_funcs.py (line ranges cited per function)
// or one pointwise block of pySHiELD/stencils/microphysics.py, with the
// operand order of the reference expression so that the same IEEE operations
// are performed (the plain form is compiled with -fmad=false).
//
// The real type R is double for the plain FP64 form. The mixed form
// instantiates the process-rate functions with R = float and keeps
// saturation adjustment, sedimentation and the budgets in double.
#pragma once

#include <cstdint>
#ifndef __CUDACC__
#include <cmath>
#include <type_traits>
#endif

#include "mp_params.h"

#ifdef __CUDACC__
#define SHD __device__ __forceinline__
// pointwise physics: also compiled for the host, where the adjoint tests
// instantiate it with a dual-number type
#define SHP __host__ __device__ __forceinline__
#else
#define SHD inline
#define SHP inline
#endif

#include "mp_math.cuh"

namespace shield {
inline namespace SHIELD_ARITH {

// microphysics_funcs.py:7-42 (numeric table kept identical)
constexpr double VCONS = 6.6280504;
constexpr double VCONG = 87.2382675;
constexpr double NORMS = 942477796.076938;
constexpr double NORMG = 5026548245.74367;
constexpr double VCONR = 2503.23638966667;
constexpr double NORMR = 25132741228.7183;
constexpr double THR = 1.0e-8;
constexpr double THI = 1.0e-8;
constexpr double THG = 1.0e-8;
constexpr double THS = 1.0e-8;
constexpr double AA = -4.14122e-5;
constexpr double BB = -0.00538922;
constexpr double CC = -0.0516344;
constexpr double DD_FS = 0.00216078;
constexpr double EE = 1.9714;
constexpr double VR_MIN = 1.0e-3;
constexpr double VF_MIN = 1.0e-5;
constexpr double P_MIN = 100.0;
constexpr double DT_FR = 8.0;
constexpr double SFCRHO = 1.2;
constexpr double RHOS = 1.0e2;
constexpr double RHOG = 4.0e2;
constexpr double RHOR = 1.0e3;
constexpr double QCMIN = 1.0e-12;
constexpr double QRMIN = 1.0e-8;
constexpr double QVMIN = 1.0e-20;

// The FP64 exp/log/pow sequences are large; called through these
// out-of-line wrappers they exist once in the kernel instead of at every one
// of their call sites, which keeps the kernel within the instruction cache.
#if defined(__CUDACC__) && !defined(SHIELD_INLINE_MATH)
#define SHIELD_MATH_ATTR static __host__ __device__ __noinline__
#elif defined(__CUDACC__)
#define SHIELD_MATH_ATTR __host__ __device__ __forceinline__
#else
#define SHIELD_MATH_ATTR static inline
#endif
SHIELD_MATH_ATTR double xexp(double x) {
#if SHIELD_FAST_FP64
  return fast_exp(x);
#else
  return exp(x);
#endif
}
SHIELD_MATH_ATTR double xlog(double x) {
#if SHIELD_FAST_FP64
  return fast_log(x);
#else
  return log(x);
#endif
}
SHIELD_MATH_ATTR double xpow(double x, double y) { return pow(x, y); }
// exp(c log x), x > 0, for a constant c
template <typename T>
SHP T xpowc(const T& x, double c) {
  return xexp(c * xlog(x));
}
SHIELD_MATH_ATTR double xpowc(double x, double c) {
#if SHIELD_FAST_FP64
  return fast_powc(x, c);
#else
  return exp(c * log(x));
#endif
}
// x^c where the reference takes a power
template <typename T>
SHP T xpowp(const T& x, double c) {
  return xpow(x, T(c));
}
SHP double xpowp(double x, double c) {
#if SHIELD_FAST_FP64
  return xpowc(x, c);
#else
  return xpow(x, c);
#endif
}

SHP double dim(double x, double y) {
  double d = x - y;
  return d > 0.0 ? d : 0.0;
}
SHP double sq(double x) { return x * x; }

// ---------------------------------------------------- microphysics_funcs.py:52-145
// wqs1 / iqs1: the saturation humidity over water / ice; wqs2 / iqs2 add its
// temperature derivative. The reference's expressions, by the types that
// have no form of their own (dual numbers, the host) and outside the
// temperatures of sat_over_t.
template <typename T>
SHP T wqs1_ref(const MpConst& K, T ta, T den) {
  return (K.E00 * xexp((K.DC_VAP * xlog(ta / K.TICE) + K.LV0 * (ta - K.TICE) / (ta * K.TICE)) / K.RVGAS)) /
         (K.RVGAS * ta * den);
}
template <typename T>
SHP T iqs1_ref(const MpConst& K, T ta, T den) {
  if (ta < K.TICE) {
    if (ta >= K.T_SAT_MIN) {
      return (K.E00 * xexp((K.D2ICE * xlog(ta / K.TICE) + K.LI2 * (ta - K.TICE) / (ta * K.TICE)) / K.RVGAS)) /
             (K.RVGAS * ta * den);
    }
    return K.iqs_lo_num / (K.RVGAS * K.T_SAT_MIN * den);
  }
  if (ta <= K.TICE + 102.0) return wqs1_ref<T>(K, ta, den);
  return wqs1_ref<T>(K, T(K.TICE + 102.0), den);
}
template <typename T>
SHP T wqs2_ref(const MpConst& K, T ta, T den, T& dqdt) {
  T tmp = wqs1_ref(K, ta, den);
  dqdt = tmp * (K.DC_VAP + K.LV0 / ta) / (K.RVGAS * ta);
  return tmp;
}
template <typename T>
SHP T iqs2_ref(const MpConst& K, T ta, T den, T& dqdt) {
  T tmp = iqs1_ref(K, ta, den);
  if (ta < K.TICE) {
    if (ta >= K.T_SAT_MIN)
      dqdt = tmp * (K.D2ICE + K.LI2 / ta) / (K.RVGAS * ta);
    else
      dqdt = tmp * (K.D2ICE + K.LI2 / K.T_SAT_MIN) / (K.RVGAS * K.T_SAT_MIN);
  } else {
    if (ta <= K.TICE + 102.0)
      dqdt = tmp * (K.DC_VAP + K.LV0 / ta) / (K.RVGAS * ta);
    else
      dqdt = tmp * (K.DC_VAP + K.LV0 / (K.TICE + 102.0)) / (K.RVGAS * (K.TICE + 102.0));
  }
  return tmp;
}
#ifdef __CUDACC__
struct QSat {
  double q, dq;
};
static __device__ __noinline__ QSat qsat_far(const MpConst& K, int ice, double ta, double den) {
  QSat r;
  r.q = ice ? iqs2_ref<double>(K, ta, den, r.dq) : wqs2_ref<double>(K, ta, den, r.dq);
  return r;
}
// One out-of-line copy serves water and ice; a level of an ice call at or
// above T0 takes the water form, as iqs1 does. 62 FP64 operations against
// about 110 and two nested calls for the reference's expression with CUDA's
// exp and log and IEEE divisions.
static __device__ __noinline__ QSat qsat_near(int ice, double ta, double den, double rden) {
  const bool i = ice && ta < PH_TICE;
  const double a = i ? PH_D2ICE / PH_RVGAS : PH_DC_VAP / PH_RVGAS;
  const double b = i ? PH_LI2 / (PH_RVGAS * PH_TICE) : PH_LV0 / (PH_RVGAS * PH_TICE);
  const double c2 = i ? PH_LI2 / PH_RVGAS : PH_LV0 / PH_RVGAS;
  if (ice) ta = ta <= PH_TICE + 102.0 ? ta : PH_TICE + 102.0;
  double r;
  QSat s;
  s.q = quot(sat_over_t(ta, PH_TICE, PH_E00 / PH_RVGAS, a, b, r), den, rden);
  s.dq = __dmul_rn(__dmul_rn(s.q, r), __fma_rn(c2, r, a));
  return s;
}
// rden: recip(den)
__device__ __forceinline__ QSat qsat(const MpConst& K, int ice, double ta, double den, double rden) {
  if (ta > QS_TLO && ta < QS_THI) return qsat_near(ice, ta, den, rden);
  return qsat_far(K, ice, ta, den);
}
#endif
template <typename T>
SHP T wqs1(const MpConst& K, T ta, T den) {
#if SHIELD_FAST_FP64
  if constexpr (std::is_same<T, double>::value) return qsat(K, 0, ta, den, recip(den)).q;
#endif
  return wqs1_ref(K, ta, den);
}
template <typename T>
SHP T wqs2(const MpConst& K, T ta, T den, T& dqdt) {
#if SHIELD_FAST_FP64
  if constexpr (std::is_same<T, double>::value) {
    const QSat s = qsat(K, 0, ta, den, recip(den));
    dqdt = s.dq;
    return s.q;
  }
#endif
  return wqs2_ref(K, ta, den, dqdt);
}
template <typename T>
SHP T iqs1(const MpConst& K, T ta, T den) {
#if SHIELD_FAST_FP64
  if constexpr (std::is_same<T, double>::value) return qsat(K, 1, ta, den, recip(den)).q;
#endif
  return iqs1_ref(K, ta, den);
}
template <typename T>
SHP T iqs2(const MpConst& K, T ta, T den, T& dqdt) {
#if SHIELD_FAST_FP64
  if constexpr (std::is_same<T, double>::value) {
    const QSat s = qsat(K, 1, ta, den, recip(den));
    dqdt = s.dq;
    return s.q;
  }
#endif
  return iqs2_ref(K, ta, den, dqdt);
}

// ---------------------------------------------------- microphysics_funcs.py:148-179
template <typename R>
SHP R acr3d(R v1, R v2, R q1, R q2, R c, R cac_ik, R cac_i1k, R cac_i2k, R rho) {
  R t1 = qsqrt(q1 * rho);
  R s1 = qsqrt(q2 * rho);
  R s2 = qsqrt(s1);
  return c * fabs(v1 - v2) * q1 * s2 * (cac_ik * t1 + cac_i1k * qsqrt(t1) * s2 + cac_i2k * s1);
}
template <typename R>
SHP R smlt(R tc, R dqs, R qsrho, R psacw, R psacr, R c_0, R c_1, R c_2, R c_3, R c_4, R rho, R rhofac) {
  return (qdiv(c_0 * tc, rho) - c_1 * dqs) * (c_2 * qsqrt(qsrho) + c_3 * xpowp(qsrho, 0.65625) * qsqrt(rhofac)) +
         c_4 * tc * (psacw + psacr);
}
template <typename R>
SHP R gmlt(R tc, R dqs, R qgrho, R pgacw, R pgacr, R c_0, R c_1, R c_2, R c_3, R c_4, R rho) {
  return (qdiv(c_0 * tc, rho) - c_1 * dqs) *
             (c_2 * qsqrt(qgrho) + qdiv(c_3 * xpowp(qgrho, 0.6875), xpowp(rho, 0.25))) +
         c_4 * tc * (pgacw + pgacr);
}

template <typename T>
SHP T cvm_of(const MpConst& K, T qv, T q_liq, T q_sol) {
  return K.c_air + qv * K.c_vap + q_liq * K.C_LIQ + q_sol * K.C_ICE;
}

// ---------------------------------------------------- microphysics_funcs.py:182-265
template <typename T>
SHP void revap_racc(const MpConst& K, double dt, double h_var, T& qg, T& qi, T& ql, T& qr, T& qs, T& qv, T& tz,
                    T den, T denfac) {
  if ((tz > K.t_wfr) && (qr > QRMIN)) {
    T lhl = K.lv00 + K.d0_vap * tz;
    T q_liq = ql + qr;
    T q_sol = qi + qs + qg;
    T cvm = cvm_of(K, qv, q_liq, q_sol);
    T lcpk = qdiv(lhl, cvm);
    T tin = tz - lcpk * ql;
    T qpz = qv + ql;
    T dqsdt;
    T qsat = wqs2(K, tin, den, dqsdt);
    T dqh = qmax(ql, h_var * qmax(qpz, QCMIN));
    dqh = qmin(dqh, 0.2 * qpz);
    T dqv = qsat - qv;
    T q_minus = qpz - dqh;
    T q_plus = qpz + dqh;
    // Evaporation needs qsat > q_minus, accretion qsat < q_minus (with the
    // rain as it came): a level does one of the two, and lanes of either kind
    // share one evaluation of their powers of the rain's density.
    const bool evaporates = (dqv > QVMIN) && (qsat > q_minus);
    const bool accretes = !evaporates && (ql > 1.0e-6) && (qsat < q_minus);
    if (evaporates || accretes) {
      const T qden = qr * den;
      const T pw = xpowc(qden, evaporates ? 0.725 : 0.95);
      if (evaporates) {
        T dq;
        if (qsat > q_plus)
          dq = qsat - qpz;
        else
          dq = qdiv(0.25 * sq(q_minus - qsat), dqh);
        T t2 = tin * tin;
        T evap = qdiv(K.crevp[0] * t2 * dq * (K.crevp[1] * qsqrt(qden) + K.crevp[2] * pw),
                      K.crevp[3] * t2 + K.crevp[4] * qsat * den);
        evap = qmin(qr, qmin(dt * evap, qdiv(dqv, 1.0 + lcpk * dqsdt)));
        qr = qr - evap;
        qv = qv + evap;
        q_liq = q_liq - evap;
        cvm = cvm_of(K, qv, q_liq, q_sol);
        tz = tz - qdiv(evap * lhl, cvm);
      } else {
        T sink = dt * denfac * K.cracw * pw;
        sink = qdiv(sink, 1.0 + sink) * ql;
        ql = ql - sink;
        qr = qr + sink;
      }
    }
  }
}

// ---------------------------------------------------- microphysics_funcs.py:268-341
template <typename T>
SHP void fall_speed(const MpConst& K, T qg, T qi, T qs, T tk, T den, T& vtg, T& vti, T& vts) {
  T rhof = qsqrt(qmin(10.0, qdiv(SFCRHO, den)));
  if (K.const_vi) {
    vti = K.vi_fac;
  } else {
    T vi0 = 0.01 * K.vi_fac;
    if (qi < THI) {
      vti = VF_MIN;
    } else {
      T tc = tk - K.tice;
      vti = (3.0 + qdivc(xlog(qi * den), K.log_10, K.r_log_10)) * (tc * (AA * tc + BB) + CC) + DD_FS * tc + EE;
      vti = vi0 * xexp(K.log_10 * vti) * 0.8;
      vti = qmin(K.vi_max, qmax(VF_MIN, vti));
    }
  }
  if (K.const_vs) {
    vts = K.vs_fac;
  } else {
    if (qs < THS) {
      vts = VF_MIN;
    } else {
      vts = K.vs_fac * VCONS * rhof * xpowc(qdivc(qs * den, NORMS, 1.0 / NORMS), 0.0625);
      vts = qmin(K.vs_max, qmax(VF_MIN, vts));
    }
  }
  if (K.const_vg) {
    vtg = K.vg_fac;
  } else {
    if (qg < THG) {
      vtg = VF_MIN;
    } else {
      vtg = K.vg_fac * VCONG * rhof * qsqrt(qsqrt(qsqrt(qdivc(qg * den, NORMG, 1.0 / NORMG))));
      vtg = qmin(K.vg_max, qmax(VF_MIN, vtg));
    }
  }
}

// microphysics_funcs.py:344-372 (the no_fall == 0 branch)
template <typename T>
SHP T rain_fspeed(const MpConst& K, T qrz, T den) {
  if (K.const_vr) return K.vr_fac;
  T qden = qrz * den;
  if (qrz < THR) return VR_MIN;
  T v = K.vr_fac * VCONR * qsqrt(qmin(10.0, qdiv(SFCRHO, den))) * xpowc(qdivc(qden, NORMR, 1.0 / NORMR), 0.2);
  return qmin(K.vr_max, qmax(VR_MIN, v));
}

// ---------------------------------------------------- microphysics_funcs.py:375-428
template <typename T>
SHP void autoconv_no_subgrid_var(const MpConst& K, T& qlz, T& qrz, T tz, T den, T ccn, T c_praut) {
  T qc0 = K.fac_rc * ccn;
  if (tz > K.t_wfr) {
    T qc = K.use_ccn ? qc0 : qdiv(qc0, den);
    T dq = qlz - qc;
    if (dq > 0.0) {
      T sink = qmin(dq, K.dt_rain * c_praut * den * xpowc(qlz, K.so3));
      qlz = qlz - sink;
      qrz = qrz + sink;
    }
  }
}
template <typename T>
SHP void autoconv_subgrid_var(const MpConst& K, T& qlz, T& qrz, T tz, T den, T ccn, T c_praut, T dl) {
  T qc0 = K.fac_rc * ccn;
  if (tz > K.t_wfr + DT_FR) {
    dl = qmin(qmax(1.0e-6, dl), 0.5 * qlz);
    T qc = K.use_ccn ? qc0 : qdiv(qc0, den);
    T dq = 0.5 * (qlz + dl - qc);
    if (dq > 0.0) {
      T sink = qmin(1.0, qdiv(dq, dl)) * K.dt_rain * c_praut * den * xpowc(qlz, K.so3);
      qlz = qlz - sink;
      qrz = qrz + sink;
    }
  }
}

// exp / log in the rate type R of subgrid_z_proc: the FP64 wrappers (and the
// dual-number overloads found by argument-dependent lookup) by default,
// single precision for R = float
template <typename R>
SHP R rexp(R x) { return xexp(x); }
template <typename R>
SHP R rlog(R x) { return xlog(x); }
template <>
SHP float rexp<float>(float x) { return expf(x); }
template <>
SHP float rlog<float>(float x) { return logf(x); }
template <typename R>
SHP R rpowc(R x, double c) { return xpowc(x, c); }
template <>
SHP float rpowc<float>(float x, double c) { return expf(float(c) * logf(x)); }
SHP float sq(float x) { return x * x; }

// The heat capacity of the saturation adjustment's latent-heat steps. The
// FP64 step divides by it at every use, as the reference does; the mixed
// form keeps its reciprocal and multiplies (FP64 either way).
template <typename T, bool RECIPROCAL>
struct HeatCap {
  Divisor<T> d;
  SHP void set(T c) { d = Divisor<T>(c); }
  SHP T div(T a) const {
#if SHIELD_FAST_FP64
    if constexpr (RECIPROCAL) return a * d.r;
#endif
    return d(a);
  }
};

// ---------------------------------------------------- microphysics_funcs.py:431-850
// R is the type of the deposition/sublimation and Bigg-freezing rate
// expressions (T for the FP64 step; float for the mixed form). Every
// saturation humidity, latent-heat temperature step and state update stays
// in T. The mixed form (R = float, which passes KF) takes the latent-heat
// steps with the heat capacity's reciprocal, still FP64.
template <typename T, typename R = T>
SHP void subgrid_z_proc(const MpConst& K, double h_var, double rh_adj, double rh_rain, T& qaz, T& qgz, T& qiz,
                        T& qlz, T& qrz, T& qsz, T& qvz, T& tz, T den, T denfac, T p1,
                        const MpConstF* KF = nullptr) {
  constexpr bool FAST = std::is_same<R, float>::value;
  const T tice = K.tice, t_wfr = K.t_wfr, t_sub = K.t_sub;
  const Divisor<T> by_den(den);
  // the saturation humidities (and derivatives) over water and ice
  auto qs_w = [&](T ta, T* dqdt) -> T {
#if SHIELD_FAST_FP64
    if constexpr (std::is_same<T, double>::value) {
      const QSat r = qsat(K, 0, ta, den, by_den.r);
      if (dqdt) *dqdt = r.dq;
      return r.q;
    }
#endif
    return dqdt ? wqs2(K, ta, den, *dqdt) : wqs1(K, ta, den);
  };
  auto qs_i = [&](T ta, T* dqdt) -> T {
#if SHIELD_FAST_FP64
    if constexpr (std::is_same<T, double>::value) {
      const QSat r = qsat(K, 1, ta, den, by_den.r);
      if (dqdt) *dqdt = r.dq;
      return r.q;
    }
#endif
    return dqdt ? iqs2(K, ta, den, *dqdt) : iqs1(K, ta, den);
  };
  HeatCap<T, FAST> H;
  // x / (tice - t_wfr): a product with the reciprocal in the mixed form
  auto over_tw = [&](T x) -> T {
    if constexpr (FAST)
      return x * KF->qs_rtw;
    else
      return qdiv(x, tice - t_wfr);
  };
  T lhl = K.lv00 + K.d0_vap * tz;
  T lhi = K.LI00 + K.DC_ICE * tz;
  T q_liq = qlz + qrz;
  T q_sol = qiz + qsz + qgz;
  H.set(cvm_of(K, qvz, q_liq, q_sol));
  T lcpk = H.div(lhl);
  T icpk = H.div(lhi);
  T tcpk = lcpk + icpk;
  T tcp3 = lcpk + icpk * qmin(1.0, over_tw(dim(tice, tz)));
  (void)tcpk;
  if (!(p1 >= P_MIN)) return;
  if (tz < K.T_MIN) {
    T sink = dim(1.0e-7, qvz);
    qvz = qvz - sink;
    qiz = qiz + sink;
    q_sol = q_sol + sink;
    H.set(cvm_of(K, qvz, q_liq, q_sol));
    tz = tz + H.div(sink * (lhl + lhi));
    if (!K.do_qa) qaz = qaz + 1.0;
    return;
  }
  lhl = K.lv00 + K.d0_vap * tz;
  lhi = K.LI00 + K.DC_ICE * tz;
  lcpk = H.div(lhl);
  icpk = H.div(lhi);
  tcpk = lcpk + icpk;
  tcp3 = lcpk + icpk * qmin(1.0, over_tw(dim(tice, tz)));
  T qpz = qvz + qlz + qiz;
  T tin = tz - qdiv(lhl * (qlz + qiz) + lhi * qiz,
                    K.c_air + qpz * K.c_vap + qrz * K.C_LIQ + (qsz + qgz) * K.C_ICE);
  bool warm = tin > t_sub + 6.0;
  if (warm) {
    bool dry;
    if constexpr (FAST)
      dry = qpz < rh_adj * qs_i(tin, nullptr);  // qs > 0: rh < rh_adj without the division
    else
      dry = qdiv(qpz, qs_i(tin, nullptr)) < rh_adj;
    if (dry) {
      tz = tin;
      qvz = qpz;
      qlz = 0.0;
      qiz = 0.0;
      return;  // the adjustment block below requires rh >= rh_adj
    }
  }
  // cloud water <-> vapour adjustment (:531-554)
  T dwsdt;
  T qsw = qs_w(tz, &dwsdt);
  T dq0 = qsw - qvz;
  T evap;
  if (dq0 > 0.0) {
    T factor = qmin(1.0, K.fac_l2v * qdiv(10.0 * dq0, qsw));
    evap = qmin(qlz, qdiv(factor * dq0, 1.0 + tcp3 * dwsdt));
  } else {
    evap = qdiv(dq0, 1.0 + tcp3 * dwsdt);
  }
  qvz = qvz + evap;
  qlz = qlz - evap;
  q_liq = q_liq - evap;
  H.set(cvm_of(K, qvz, q_liq, q_sol));
  tz = tz - H.div(evap * lhl);
  lhi = K.LI00 + K.DC_ICE * tz;
  icpk = H.div(lhi);
  // forced freezing below t_wfr (:560-575)
  T dtmp = t_wfr - tz;
  if ((dtmp > 0.0) && (qlz > QCMIN)) {
    T sink = qmin(qlz, qmin(qlz * dtmp * 0.125, qdiv(dtmp, icpk)));
    qlz = qlz - sink;
    qiz = qiz + sink;
    q_liq = q_liq - sink;
    q_sol = q_sol + sink;
    H.set(cvm_of(K, qvz, q_liq, q_sol));
    tz = tz + H.div(sink * lhi);
  }
  lhi = K.LI00 + K.DC_ICE * tz;
  icpk = H.div(lhi);
  // Bigg mechanism (:581-605)
  T dt_pisub;
  if (K.fast_sat_adj) {
    dt_pisub = 0.5 * K.dts;
  } else {
    dt_pisub = K.dts;
    T tc = tice - tz;
    if ((qlz > QRMIN) && (tc > 0.0)) {
      T sink = T(R(3.3333e-10) * R(K.dts) * (rexp(R(0.66) * R(tc)) - R(1.0)) * R(den) * R(qlz) * R(qlz));
      sink = qmin(qlz, qmin(qdiv(tc, icpk), sink));
      qlz = qlz - sink;
      qiz = qiz + sink;
      q_liq = q_liq - sink;
      q_sol = q_sol + sink;
      H.set(cvm_of(K, qvz, q_liq, q_sol));
      tz = tz + H.div(sink * lhi);
    }
  }
  lhl = K.lv00 + K.d0_vap * tz;
  lhi = K.LI00 + K.DC_ICE * tz;
  lcpk = H.div(lhl);
  icpk = H.div(lhi);
  tcpk = lcpk + icpk;
  // ice deposition / sublimation (:614-661)
  if (tz < tice) {
    T dqsdt;
    T qsi = qs_i(tz, &dqsdt);
    T dq = qvz - qsi;
    T sink = qdiv(dq, 1.0 + tcpk * dqsdt);
    T pidep;
    if (qiz > QRMIN) {
      pidep = T(qdiv(R(dt_pisub) * R(dq) * R(349138.78) * rpowc(R(qiz) * R(den), 0.875),
                     qdiv(R(qsi) * R(den) * R(K.LAT2), R(0.0243) * R(K.RVGAS) * sq(R(tz))) + R(4.42478e4)));
    } else {
      pidep = 0.0;
    }
    if (dq > 0.0) {
      T tmp = tice - tz;
      T qi_crt = K.qi_gen * qmin(K.qi_lim, 0.1 * tmp);
      qi_crt = by_den(qi_crt);
      sink = qmin(sink, qmin(qmax(qi_crt - qiz, pidep), qdiv(tmp, tcpk)));
    } else {
      pidep = pidep * qmin(1.0, dim(tz, t_sub) * 0.2);
      sink = qmax(pidep, qmax(sink, -qiz));
    }
    qvz = qvz - sink;
    qiz = qiz + sink;
    q_sol = q_sol + sink;
    H.set(cvm_of(K, qvz, q_liq, q_sol));
    tz = tz + H.div(sink * (lhl + lhi));
  }
  lhl = K.lv00 + K.d0_vap * tz;
  lhi = K.LI00 + K.DC_ICE * tz;
  lcpk = H.div(lhl);
  icpk = H.div(lhi);
  tcpk = lcpk + icpk;
  // snow sublimation / deposition (:670-706)
  if (qsz > QRMIN) {
    T dqsdt;
    T qsi = qs_i(tz, &dqsdt);
    T qden = qsz * den;
    const R qdr = R(qden);
    const R tmp = rpowc(qdr, 0.65625);
    T tsq = tz * tz;
    T dq = qdiv(qsi - qvz, 1.0 + tcpk * dqsdt);
    const R tsr = R(tsq);
    T pssub = T(qdiv(R(K.cssub[0]) * tsr * (R(K.cssub[1]) * qsqrt(qdr) + R(K.cssub[2]) * tmp * qsqrt(R(denfac))),
                     R(K.cssub[3]) * tsr + R(K.cssub[4]) * R(qsi) * R(den)));
    pssub = (qsi - qvz) * K.dts * pssub;
    if (pssub > 0.0) {
      pssub = qmin(pssub * qmin(1.0, dim(tz, t_sub) * 0.2), qsz);
    } else {
      if (tz > tice)
        pssub = 0.0;
      else
        pssub = qmax(pssub, qmax(dq, qdiv(tz - tice, tcpk)));
    }
    qsz = qsz - pssub;
    qvz = qvz + pssub;
    q_sol = q_sol - pssub;
    H.set(cvm_of(K, qvz, q_liq, q_sol));
    tz = tz - H.div(pssub * (lhl + lhi));
  }
  lhl = K.lv00 + K.d0_vap * tz;
  lhi = K.LI00 + K.DC_ICE * tz;
  lcpk = H.div(lhl);
  icpk = H.div(lhi);
  tcpk = lcpk + icpk;
  // graupel sublimation / deposition (:715-746)
  if (qgz > QRMIN) {
    T dqsdt;
    T qsi = qs_i(tz, &dqsdt);
    T dq = qdiv(qvz - qsi, 1.0 + tcpk * dqsdt);
    T pgsub = (qdiv(qvz, qsi) - 1.0) * qgz;
    if (pgsub > 0.0) {
      if (tz > tice)
        pgsub = 0.0;
      else
        pgsub = qmin(qmin(K.fac_v2g * pgsub, 0.2 * dq), qmin(qlz + qrz, qdiv(tice - tz, tcpk)));
    } else {
      pgsub = qmax(K.fac_g2v * pgsub, dq) * qmin(1.0, dim(tz, t_sub) * 0.1);
    }
    qgz = qgz + pgsub;
    qvz = qvz - pgsub;
    q_sol = q_sol + pgsub;
    H.set(cvm_of(K, qvz, q_liq, q_sol));
    tz = tz + H.div(pgsub * (lhl + lhi));
  }
  // minimum evaporation of rain (:751-769)
  lhl = K.lv00 + K.d0_vap * tz;
  lcpk = H.div(lhl);
  if (qrz > QCMIN) {
    T dqsdt;
    T qsw2 = qs_w(tz, &dqsdt);
    T sink = qmin(qrz, qdiv(dim(rh_rain * qsw2, qvz), 1.0 + lcpk * dqsdt));
    qvz = qvz + sink;
    qrz = qrz - sink;
    q_liq = q_liq - sink;
    H.set(cvm_of(K, qvz, q_liq, q_sol));
    tz = tz - H.div(sink * lhl);
  }
  // cloud fraction (:774-848)
  lhl = K.lv00 + K.d0_vap * tz;
  H.set(K.c_air + (qvz + q_liq + q_sol) * K.c_vap);
  lcpk = H.div(lhl);
  if (!K.do_qa) {
    q_sol = K.rad_snow ? qiz + qsz : qiz;
    q_liq = K.rad_rain ? qlz + qrz : qlz;
    T q_cond = q_liq + q_sol;
    T qpz2 = qvz + q_cond;
    T tin2 = tz - (lcpk * q_cond + icpk * q_sol);
    T qstar;
    if (tin2 <= t_wfr) {
      qstar = qs_i(tin2, nullptr);
    } else if (tin2 >= tice) {
      qstar = qs_w(tin2, nullptr);
    } else {
      T qsi = qs_i(tin2, nullptr);
      T qsw3 = qs_w(tin2, nullptr);
      T rqi;
      if (q_cond > 3.0e-6)
        rqi = qdiv(q_sol, q_cond);
      else
        rqi = over_tw(tice - tin2);
      qstar = rqi * qsi + (1.0 - rqi) * qsw3;
    }
    if (qpz2 > QRMIN) {
      T dq = qmax(QCMIN, h_var * qpz2);
      T q_plus = qpz2 + dq;
      T q_minus = qpz2 - dq;
      if (qstar < q_minus)
        qaz = qaz + 1.0;
      else if ((qstar < q_plus) && (q_cond > K.qc_crt))
        qaz = qaz + qdiv(q_plus - qstar, dq + dq);
    }
  }
}

// ---------------------------------------------------- microphysics_funcs.py:853-1227
// Ice-phase processes before the saturation adjustment; the caller runs
// subgrid_z_proc afterwards (icloud_main's tail call, :1229-1258).
template <typename T>
SHP void icloud_processes(const MpConst& K, T& qgz, T& qiz, T& qlz, T& qrz, T& qsz, T qvz, T& tz, T den, T denfac,
                          T vtgz, T vtrz, T vtsz, T p1, T di, T q_liq, T q_sol, T cvm) {
  const T tice = K.tice, dts = K.dts, rdts = K.rdts;
  T lhi = K.LI00 + K.DC_ICE * tz;
  T icpk = qdiv(lhi, cvm);
  if (!(p1 >= P_MIN)) return;
  T pgacr = 0.0;
  T pgacw = 0.0;
  T tc = tz - tice;
  if (tc >= 0.0) {
    T dqs0 = qdiv(K.ces0, p1) - qvz;
    if (qsz > QCMIN) {
      T psacw, psacr, pracs;
      if (qlz > QRMIN) {
        T factor = denfac * K.csacw * xpowc(qsz * den, 0.8125);
        psacw = qdiv(factor, 1.0 + dts * factor) * qlz;
      } else {
        psacw = 0.0;
      }
      if (qrz > QRMIN) {
        psacr = qmin(acr3d<T>(vtsz, vtrz, qrz, qsz, K.csacr, K.acco[0][1], K.acco[1][1], K.acco[2][1], den),
                     qrz * rdts);
        pracs = acr3d<T>(vtrz, vtsz, qsz, qrz, K.cracs, K.acco[0][0], K.acco[1][0], K.acco[2][0], den);
      } else {
        psacr = 0.0;
        pracs = 0.0;
      }
      T psmlt = qmax(0.0, smlt<T>(tc, dqs0, qsz * den, psacw, psacr, K.csmlt[0], K.csmlt[1], K.csmlt[2],
                                             K.csmlt[3], K.csmlt[4], den, denfac));
      T sink = qmin(qsz, qmin(dts * (psmlt + pracs), qdiv(tc, icpk)));
      qsz = qsz - sink;
      T tmp = qmin(sink, dim(K.qs_mlt, qlz));
      qlz = qlz + tmp;
      qrz = qrz + sink - tmp;
      q_liq = q_liq + sink;
      q_sol = q_sol - sink;
      cvm = cvm_of(K, qvz, q_liq, q_sol);
      tz = tz - qdiv(sink * lhi, cvm);
      tc = tz - tice;
    }
    lhi = K.LI00 + K.DC_ICE * tz;
    icpk = qdiv(lhi, cvm);
    if ((qgz > QCMIN) && (tc > 0.0)) {
      if (qrz > QRMIN) {
        pgacr = qmin(acr3d<T>(vtgz, vtrz, qrz, qgz, K.cgacr, K.acco[0][2], K.acco[1][2], K.acco[2][2], den),
                     rdts * qrz);
      }
      T qden = qgz * den;
      if (qlz > QRMIN) {
        T factor = qdiv(K.cgacw * qden, qsqrt(den * qsqrt(qsqrt(qden))));
        pgacw = qdiv(factor, 1.0 + dts * factor) * qlz;
      }
      T pgmlt = dts * gmlt<T>(tc, dqs0, qden, pgacw, pgacr, K.cgmlt[0], K.cgmlt[1], K.cgmlt[2],
                                        K.cgmlt[3], K.cgmlt[4], den);
      pgmlt = qmin(qmax(0.0, pgmlt), qmin(qgz, qdiv(tc, icpk)));
      qgz = qgz - pgmlt;
      qrz = qrz + pgmlt;
      q_liq = q_liq + pgmlt;
      q_sol = q_sol - pgmlt;
      cvm = cvm_of(K, qvz, q_liq, q_sol);
      tz = tz - qdiv(pgmlt * lhi, cvm);
    }
  } else {
    if (qiz > 3.0e-7) {
      T psaci;
      if (qsz > 1.0e-7) {
        T factor = dts * denfac * K.csaci * xexp(0.05 * tc + 0.8125 * xlog(qsz * den));
        psaci = qdiv(factor, 1.0 + factor) * qiz;
      } else {
        psaci = 0.0;
      }
      T qim = qdiv(K.qi0_crt, den);
      T tmp = K.const_vi ? K.fac_i2s : K.fac_i2s * xexp(0.025 * tc);
      di = qmax(di, QRMIN);
      T q_plus = qiz + di;
      T psaut;
      if (q_plus > (qim + QRMIN)) {
        T dq;
        if (qim > (qiz - di))
          dq = qdiv(0.25 * sq(q_plus - qim), di);
        else
          dq = qiz - qim;
        psaut = tmp * dq;
      } else {
        psaut = 0.0;
      }
      T sink = qmin(0.75 * qiz, psaci + psaut);
      qiz = qiz - sink;
      qsz = qsz + sink;
      if (qgz > 1.0e-6) {
        T factor = dts * K.cgaci * qsqrt(den) * qgz;
        T pgaci = qdiv(factor, 1.0 + factor) * qiz;
        qiz = qiz - pgaci;
        qgz = qgz + pgaci;
      }
    }
    tc = tz - tice;
    if ((qrz > 1e-7) && (tc < 0.0)) {
      T psacr;
      if (qsz > 1.0e-7)
        psacr = dts * acr3d<T>(vtsz, vtrz, qrz, qsz, K.csacr, K.acco[0][1], K.acco[1][1], K.acco[2][1], den);
      else
        psacr = 0.0;
      T pgfr = qdiv(dts * K.cgfr[0], den) * (xexp(-K.cgfr[1] * tc) - 1.0) * xpowc(qrz * den, 1.75);
      T sink = psacr + pgfr;
      T factor = qdiv(qmin(sink, qmin(qrz, qdiv(-tc, icpk))), qmax(sink, QRMIN));
      psacr = factor * psacr;
      pgfr = factor * pgfr;
      sink = psacr + pgfr;
      qrz = qrz - sink;
      qsz = qsz + psacr;
      qgz = qgz + pgfr;
      q_liq = q_liq - sink;
      q_sol = q_sol + sink;
      cvm = cvm_of(K, qvz, q_liq, q_sol);
      tz = tz + qdiv(sink * lhi, cvm);
    }
    lhi = K.LI00 + K.DC_ICE * tz;
    icpk = qdiv(lhi, cvm);
    if (qsz > 1.0e-7) {
      T sink;
      if (qgz > QRMIN)
        sink = dts * acr3d<T>(vtgz, vtsz, qsz, qgz, K.cgacs, K.acco[0][3], K.acco[1][3], K.acco[2][3], den);
      else
        sink = 0.0;
      T qsm = qdiv(K.qs0_crt, den);
      if (qsz > qsm) {
        T factor = dts * 1.0e-3 * xexp(0.09 * (tz - tice));
        sink = sink + qdiv(factor, 1.0 + factor) * (qsz - qsm);
      }
      sink = qmin(qsz, sink);
      qsz = qsz - sink;
      qgz = qgz + sink;
    }
    if ((qgz > 1.0e-7) && (tz < K.tice0)) {
      if (qlz > 1.0e-6) {
        T qden = qgz * den;
        T factor = qdiv(dts * K.cgacw * qden, qsqrt(den * qsqrt(qsqrt(qden))));
        pgacw = qdiv(factor, 1.0 + factor) * qlz;
      } else {
        pgacw = 0.0;
      }
      if (qrz > 1.0e-6) {
        pgacr = qmin(dts * acr3d<T>(vtgz, vtrz, qrz, qgz, K.cgacr, K.acco[0][2], K.acco[1][2], K.acco[2][2], den),
                     qrz);
      } else {
        pgacr = 0.0;
      }
      T sink = pgacr + pgacw;
      T factor = qdiv(qmin(sink, qdiv(dim(tice, tz), icpk)), qmax(sink, QRMIN));
      pgacr = factor * pgacr;
      pgacw = factor * pgacw;
      sink = pgacr + pgacw;
      qgz = qgz + sink;
      qrz = qrz - pgacr;
      qlz = qlz - pgacw;
      q_liq = q_liq - sink;
      q_sol = q_sol + sink;
      cvm = cvm_of(K, qvz, q_liq, q_sol);
      tz = tz + qdiv(sink * lhi, cvm);
    }
  }
}

// -------------------------------------- pointwise blocks of the step body
// Cloud ice melting at and below the first level warmer than tice, at the
// start of sedimentation (microphysics.py:706-746).
template <typename T>
SHP void sedi_ice_melt(const MpConst& K, T qv, T& ql, T& qr, T& qi, T qs, T qg, T& tz) {
  const T lhi = K.LI00 + K.DC_ICE * tz;
  T q_liq = ql + qr;
  T q_sol = qi + qs + qg;
  T cvm = K.c_air + qv * K.c_vap + q_liq * K.C_LIQ + q_sol * K.C_ICE;
  const T icpk = qdiv(lhi, cvm);
  const T tc = tz - K.tice;
  if ((qi > QCMIN) && (tc > 0.0)) {
    const T sink = qmin(qi, qdiv(K.fac_imlt * tc, icpk));
    const T tmp = qmin(sink, dim(K.ql_mlt, ql));
    ql = ql + tmp;
    qr = qr + sink - tmp;
    qi = qi - sink;
    q_liq = q_liq + sink;
    q_sol = q_sol - sink;
    cvm = K.c_air + qv * K.c_vap + q_liq * K.C_LIQ + q_sol * K.C_ICE;
    tz = tz - qdiv(sink * lhi, cvm);
  }
}

// Instant melting of cloud ice above tice, or freezing of cloud water below
// t_wfr, at the start of icloud (microphysics.py:1298-1339); returns the
// liquid and solid totals and cvm that icloud_processes starts from.
template <typename T>
SHP void icloud_melt_freeze(const MpConst& K, T qv, T& ql, T& qr, T& qi, T& qs, T qg, T& tz, T den, T& q_liq,
                            T& q_sol, T& cvm) {
  const T lhi = K.LI00 + K.DC_ICE * tz;
  q_liq = ql + qr;
  q_sol = qi + qs + qg;
  cvm = K.c_air + qv * K.c_vap + q_liq * K.C_LIQ + q_sol * K.C_ICE;
  const T icpk = qdiv(lhi, cvm);
  if ((tz > K.tice) && (qi > QCMIN)) {
    const T melt = qmin(qi, qdiv(K.fac_imlt * (tz - K.tice), icpk));
    const T tmp = qmin(melt, dim(K.ql_mlt, ql));
    ql = ql + tmp;
    qr = qr + melt - tmp;
    qi = qi - melt;
    q_liq = q_liq + melt;
    q_sol = q_sol - melt;
    cvm = K.c_air + qv * K.c_vap + q_liq * K.C_LIQ + q_sol * K.C_ICE;
    tz = tz - qdiv(melt * lhi, cvm);
  } else if ((tz < K.t_wfr) && (ql > QCMIN)) {
    const T dtmp = K.t_wfr - tz;
    const T factor = qmin(1.0, dtmp / DT_FR);  // exact: DT_FR is a power of two
    const T sink = qmin(ql * factor, qdiv(dtmp, icpk));
    const T qi_crt = qdiv(K.qi_gen * qmin(K.qi_lim, 0.1 * (K.tice - tz)), den);
    const T tmp = qmin(sink, dim(qi_crt, qi));
    ql = ql - sink;
    qs = qs + sink - tmp;
    qi = qi + tmp;
    q_liq = q_liq - sink;
    q_sol = q_sol + sink;
    cvm = K.c_air + qv * K.c_vap + q_liq * K.C_LIQ + q_sol * K.C_ICE;
    tz = tz + qdiv(sink * lhi, cvm);
  }
}

// The pointwise part of fix_negative (microphysics.py:202-240): negative
// species borrow from the next one in the chain ice -> snow -> graupel ->
// rain -> cloud water -> vapour, with the latent heat.
template <typename T>
SHP void fix_negative_point(const MpConst& K, T& qv, T& ql, T& qr, T& qi, T& qs, T& qg, T& tz) {
  const T cvm = K.c_air + qv * K.c_vap + (qr + ql) * K.C_LIQ + (qi + qs + qg) * K.C_ICE;
  const Divisor<T> by_cvm(cvm);
  const T lcpk = by_cvm(K.lv00 + K.d0_vap * tz);
  const T icpk = by_cvm(K.LI00 + K.DC_ICE * tz);
  if (qi < 0.0) {
    qs = qs + qi;
    qi = 0.0;
  }
  if (qs < 0.0) {
    qg = qg + qs;
    qs = 0.0;
  }
  if (qg < 0.0) {
    qr = qr + qg;
    tz = tz - qg * icpk;
    qg = 0.0;
  }
  if (qr < 0.0) {
    ql = ql + qr;
    qr = 0.0;
  }
  if (ql < 0.0) {
    qv = qv + ql;
    tz = tz - ql * lcpk;
    ql = 0.0;
  }
}

}  // namespace SHIELD_ARITH
}  // namespace shield
