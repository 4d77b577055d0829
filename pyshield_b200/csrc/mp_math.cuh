// FP64 division, square root, exponential, logarithm and powers of the
// microphysics step, on the device.
//
// The step meets about 200 divisions and square roots and 50 exponentials
// and logarithms per level. With the general forms, most of the step's
// instructions were not its arithmetic but theirs: range checks, branches to
// a slow path, 64-bit literal coefficients built in pairs of moves (ncu, C48
// L79: 490 M warp instructions, 140 M of them FP64; with these forms, when
// they came in, 307 M and 102 M, and the C96 L79 step 3.61 -> 2.14 ms, mixed
// 2.29 -> 1.63 ms). Exp, log, powers and the humidity over ice were less
// accurate than the functions replaced then; carrying the roundings that
// mends it took 1.82 -> 1.87 ms, mixed 1.38 -> 1.39. The forms here drop what
// the step's operands do not need:
//  * divisors are finite and normal (temperatures, densities, heat
//    capacities, thicknesses, humidities), so a reciprocal is the hardware's
//    approximation and one step of the cubic Newton iteration
//    r' = r + r (e + e^2), e = 1 - b r, and a quotient is Markstein's
//    q + (a - b q) r (IBM J. Res. Dev. 34, 1990). A zero, infinite or
//    subnormal divisor gives a NaN. The quotient is the correctly rounded one
//    but for some that lie within 1e-15 units of a midpoint between two numbers
//    (none of 4e7 random operands, 14 of 5e6 made to lie there); in a
//    SHIELD_IEEE unit it is for all. A divisor used several times shares its
//    reciprocal;
//  * square roots of values >= 0 by Goldschmidt's coupled iteration on the
//    hardware's reciprocal square root, with the residual x - g^2 taken
//    exactly at the end (2 of 1.2e9 differed from the rounded root);
//  * exp and log reduce by powers of two and evaluate minimax polynomials
//    (computed for this file by Remez exchange in 60 digits; the errors are
//    noted beside them), whose coefficients are constant-bank operands; an
//    argument out of their range takes CUDA's function. exp and log carry the
//    rounding of their leading terms, and a power that of its exponent: none
//    is further off than the CUDA function in its place.
// A unit that defines SHIELD_IEEE keeps the rounding of every operation of
// the reference's expressions (CUDA's exp, log, pow and square root, quotients as
// IEEE division rounds them): see mp_ieee.cu. On the host (the adjoint tests' harness)
// and for any type but double the names are the plain operators and library
// functions.
#pragma once

namespace shield {
inline namespace SHIELD_ARITH {

#if defined(__CUDA_ARCH__)
#define SHIELD_DEVICE_FP64 1
#else
#define SHIELD_DEVICE_FP64 0
#endif
#if SHIELD_DEVICE_FP64 && !defined(SHIELD_IEEE)
#define SHIELD_FAST_FP64 1
#else
#define SHIELD_FAST_FP64 0
#endif

#ifdef __CUDACC__
// (e^r - 1 - r) / r^2 on |r| <= ln 2 / 2, degree 9 (3.6e-18 of e^r)
static __constant__ double EXPQ_C[10] = {
    0.500000000000001061676,    0.166666666666664127699,    0.04166666666653026584,      0.00833333333349433727524,
    0.0013888888943597743,      0.000198412695067695883869, 0.0000248014931361361384094, 0.00000275575862760101766395,
    2.76302339374682250928e-7,  2.50000690936568463792e-8};
// (2^r - 1) / r on |r| <= 1/2, degree 10 (3.4e-18)
static __constant__ double EXP2_C[11] = {
    0.693147180559945325805,   0.240226506959101312602,   0.0555041086648200832261,  0.00961812910759412007516,
    0.00133335581467746208208, 0.000154035304571121010251, 0.0000152527334931271240257, 0.000001321543528230637037,
    1.01781995720268829334e-7, 7.0737832484981793467e-9,  4.43477126654816555124e-10};
// (2 atanh(s) / s - 2) / s^2 in z = s^2, sqrt(1/2) <= m < sqrt(2), s = (m - 1) / (m + 1), degree 7 (1.6e-20 of log m / s)
static __constant__ double LOG_C[8] = {0.666666666666666609796, 0.400000000000062424342, 0.28571428569087348774,
                                       0.222222226465718982078, 0.181817756837742750264, 0.153870899487081287653,
                                       0.132501365763733722032, 0.132511596952031750849};
#endif

// ------------------------------------------------------- minimum and maximum
// A compare and a select; fmin and fmax also order a NaN below every number,
// which costs twice the instructions. A NaN second operand is returned, so
// that it reaches the step's check of its outputs.
template <typename A, typename B>
SHP auto qmin(const A& a, const B& b) -> decltype(fmin(a, b)) {
  return fmin(a, b);
}
template <typename A, typename B>
SHP auto qmax(const A& a, const B& b) -> decltype(fmax(a, b)) {
  return fmax(a, b);
}
SHP double qmin(double a, double b) { return a <= b ? a : b; }
SHP double qmax(double a, double b) { return a >= b ? a : b; }

// ---------------------------------------------------------------- division
#ifdef __CUDACC__
// 1 / b of a finite, normal b, within one unit in the last place. e + e^2
// rounds up, so that a b of all ones gets the upper of the two numbers its
// reciprocal lies between (1 / (2 - 2^-52) = 1/2 + 2^-54 + 2^-107, just above
// their midpoint; rounded to nearest, e + e^2 would lose the last term).
// With SHIELD_IEEE one Newton step more gives the correctly rounded 1 / b:
// from within a unit it does for every other b (Markstein 1990).
__device__ __forceinline__ double recip(double b) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  const double e = __fma_rn(-b, r, 1.0);
  r = __fma_rn(r, __fma_ru(e, e, e), r);
#ifdef SHIELD_IEEE
  r = __fma_rn(r, __fma_rn(-b, r, 1.0), r);
#endif
  return r;
}
// a / b given r = recip(b), for a normal quotient. With r correctly rounded,
// so is the quotient: its residual a - b q is exact, and r's error moves it
// by less than a quotient's distance from the nearest midpoint.
__device__ __forceinline__ double quot(double a, double b, double r) {
  const double q = __dmul_rn(a, r);
  return __fma_rn(__fma_rn(-b, q, a), r, q);
}
__device__ __forceinline__ double root(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double g = __dmul_rn(x, y);
  const double h0 = __dmul_rn(0.5, y);
  const double e = __fma_rn(-h0, g, 0.5);
  g = __fma_rn(g, e, g);
  const double h = __fma_rn(h0, e, h0);
  const double s = __fma_rn(__fma_rn(-g, g, x), h, g);
  return x == 0.0 ? x : s;  // the reciprocal root of zero is infinite
}
#endif

template <typename A, typename B>
SHP auto qdiv(const A& a, const B& b) -> decltype(a / b) {
  return a / b;
}
SHP double qdiv(double a, double b) {
#if SHIELD_DEVICE_FP64
  return quot(a, b, recip(b));
#else
  return a / b;
#endif
}
template <typename T>
SHP T qsqrt(const T& x) {
  return sqrt(x);
}
SHP double qsqrt(double x) {
#if SHIELD_FAST_FP64
  return root(x);
#else
  return sqrt(x);
#endif
}

// a / c for a constant c whose reciprocal rc the compiler or the host formed
template <typename T>
SHP T qdivc(const T& a, double c, double rc) {
  return a / c;
}
SHP double qdivc(double a, double c, double rc) {
#if SHIELD_DEVICE_FP64
  return quot(a, c, rc);
#else
  return a / c;
#endif
}

// A divisor used several times: its reciprocal is formed once.
template <typename T>
struct Divisor {
  T b;
  SHP Divisor() {}
  SHP explicit Divisor(const T& x) : b(x) {}
  SHP T operator()(const T& a) const { return a / b; }
};
template <>
struct Divisor<double> {
  double b, r;
  SHP Divisor() {}
  SHP explicit Divisor(double x) : b(x) {
#if SHIELD_DEVICE_FP64
    r = recip(x);
#else
    r = 0.0;
#endif
  }
  SHP double operator()(double a) const {
#if SHIELD_DEVICE_FP64
    return quot(a, b, r);
#else
    return a / b;
#endif
  }
};

// --------------------------------------------------------- exp, log, powers
#ifdef __CUDACC__
// p(r) of 11 coefficients, two interleaved half-length Horner chains
__device__ __forceinline__ double poly11(const double* c, double r) {
  const double r2 = __dmul_rn(r, r);
  double e = c[10], o = c[9];
#pragma unroll
  for (int n = 4; n >= 0; --n) {
    e = __fma_rn(e, r2, c[2 * n]);
    if (n > 0) o = __fma_rn(o, r2, c[2 * n - 1]);
  }
  return __fma_rn(o, r, e);
}
__device__ __forceinline__ double poly10(const double* c, double r) {
  const double r2 = __dmul_rn(r, r);
  double e = c[8], o = c[9];
#pragma unroll
  for (int n = 3; n >= 0; --n) {
    e = __fma_rn(e, r2, c[2 * n]);
    o = __fma_rn(o, r2, c[2 * n + 1]);
  }
  return __fma_rn(o, r, e);
}
// x 2^k, for a result in the normal range
__device__ __forceinline__ double scale2(double x, int k) {
  return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
}
constexpr double ROUND_MAGIC = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer in the low word

// ln 2 to 21 bits, so that a multiple of up to 2^31 is exact, and the rest
constexpr double LN2_HI = 0.6931467056274414, LN2_LO = 0.0000004749325039031672321214582;

// e^x, |x| < 700. The reduced argument x - k ln 2 (Cody and Waite's two-part
// reduction) is kept in two parts r + rl, and 1 + r with the rounding of its
// sum: 0.71 units in the last place at most, 0.290 in the mean square (CUDA's
// exp 0.87 and 0.302; the plain 1 + r P(r) 1.24 and 0.317).
__device__ __forceinline__ double exp_reduced(double x) {
  const double t = __fma_rn(x, 1.44269504088896340736, ROUND_MAGIC);
  const double kd = __dadd_rn(t, -ROUND_MAGIC);
  const double h = __fma_rn(kd, -LN2_HI, x);
  const double r = __fma_rn(kd, -LN2_LO, h);
  const double rl = __fma_rn(kd, -LN2_LO, __dadd_rn(h, -r));
  const double w = __fma_rn(__dmul_rn(r, r), poly10(EXPQ_C, r), __fma_rn(rl, r, rl));
  const double y = __dadd_rn(1.0, r);
  return scale2(__dadd_rn(y, __dadd_rn(__dadd_rn(__dadd_rn(1.0, -y), r), w)), __double2loint(t));
}
__device__ __forceinline__ double fast_exp(double x) {
  if (!(fabs(x) < 700.0)) return exp(x);
  return exp_reduced(x);
}
// x = 2^k m: k, s = (m - 1) / (m + 1) with sl, the rounding of its quotient
// and of m + 1, and 2 (atanh(s) - s), which is log m less 2 (s + sl). x
// positive, finite, normal.
struct LogParts {
  double k, s, sl, t;
};
__device__ __forceinline__ LogParts log_parts(double x) {
  const int hi = __double2hiint(x);
  const int k = (hi - 0x3fe6a09e) >> 20;  // m in [sqrt(1/2), sqrt(2))
  const double m = __hiloint2double(hi - (k << 20), __double2loint(x));
  const double f = __dadd_rn(m, -1.0);
  const double d = __dadd_rn(m, 1.0), dl = __dadd_rn(m, -__dadd_rn(d, -1.0));
  const double rd = recip(d);
  LogParts P;
  P.k = __int2double_rn(k);
  P.s = __dmul_rn(f, rd);
  P.sl = __dmul_rn(__fma_rn(-P.s, dl, __fma_rn(-P.s, d, f)), rd);
  const double z = __fma_rn(__dadd_rn(P.s, P.s), P.sl, __dmul_rn(P.s, P.s));
  const double z2 = __dmul_rn(z, z);
  double e = __fma_rn(LOG_C[6], z2, LOG_C[4]), o = __fma_rn(LOG_C[7], z2, LOG_C[5]);
  e = __fma_rn(e, z2, LOG_C[2]);
  o = __fma_rn(o, z2, LOG_C[3]);
  e = __fma_rn(e, z2, LOG_C[0]);
  o = __fma_rn(o, z2, LOG_C[1]);
  P.t = __dmul_rn(__dmul_rn(P.s, z), __fma_rn(o, z, e));
  return P;
}
// log x = h + l, l the rounding of h: k ln 2 is exact in its leading part
// and no smaller than 2 s, so the sums' roundings are
__device__ __forceinline__ double log_sum(const LogParts& P, double& l) {
  const double a = __dmul_rn(P.k, LN2_HI), b = __dadd_rn(P.s, P.s);
  const double c = __dadd_rn(a, b);
  const double t = __dadd_rn(__dadd_rn(__dadd_rn(a, -c), b),
                             __fma_rn(P.k, LN2_LO, __dadd_rn(__dadd_rn(P.sl, P.sl), P.t)));
  const double h = __dadd_rn(c, t);
  l = __dadd_rn(__dadd_rn(c, -h), t);
  return h;
}
__device__ __forceinline__ bool log_in_range(double x) {
  return (unsigned)(__double2hiint(x) - 0x00100000) < 0x7fe00000u;  // positive, normal, finite
}
// 0.53 units in the last place at most (CUDA's log 0.55, the plain sum 2.0)
__device__ __forceinline__ double fast_log(double x) {
  if (!log_in_range(x)) return log(x);
  double l;
  return log_sum(log_parts(x), l);
}
// x^c, x > 0: 2^(c log2 x). log x, log2 x and its product with c are kept in
// two parts: 1.27 units in the last place at most, 0.32 in the mean square
// (CUDA's pow 1.35 and 0.41; exp(c log x) rounds the exponent: up to
// |c log x| units). The exponential's reduced argument in two parts as well
// gives 0.71 and 0.291, and 3 % more of the step's time.
__device__ __forceinline__ double fast_powc(double x, double c) {
  if (!log_in_range(x)) return pow(x, c);
  const LogParts P = log_parts(x);
  const double l = __dadd_rn(P.s, P.s), ll = __dadd_rn(__dadd_rn(P.sl, P.sl), P.t);
  const double h = __fma_rn(l, 1.44269504088896340736, P.k);
  const double hl = __fma_rn(ll, 1.44269504088896340736, __fma_rn(l, 1.44269504088896340736, __dadd_rn(P.k, -h)));
  const double y = __dmul_rn(c, h);
  const double yl = __fma_rn(c, hl, __fma_rn(c, h, -y));
  if (!(fabs(y) < 1000.0)) return pow(x, c);
  const double t = __dadd_rn(y, ROUND_MAGIC);
  const int n = __double2loint(t);
  const double r = __dadd_rn(__dadd_rn(y, -__dadd_rn(t, -ROUND_MAGIC)), yl);
  return scale2(__fma_rn(r, poly11(EXP2_C, r), 1.0), n);
}

// The saturation vapour pressure over water or ice, e(T) = E00 exp((Dc ln(T /
// T0) + L (T - T0) / (T T0)) / Rv) for QS_TLO < T < QS_THI: with s =
// (T - T0) / (T + T0), ln(T / T0) = 2 atanh(s), whose series in z = s^2
// needs degree 8 there (minimax, 5.7e-18 of ln / s). (T - T0) / T, which
// reaches -0.8 and meets a factor of 23 to 25, is the rounded quotient: as
// (T - T0) (1 / T), with 1 / T and 1 / (T + T0) from one reciprocal of their
// product, the humidity over ice was further off than the reference's
// expression with CUDA's functions (170 to 330 K: 6.7e-16 in the mean square
// and 5.3e-15 at most, against 6.4e-16 and 4.8e-15; now 5.3e-16 and 3.1e-15).
// Returns e(T) / T and 1 / T.
static __constant__ double ATANH_C[9] = {0.66666666666667514115,  0.399999999996019593816, 0.285714286357600045542,
                                         0.222222171320237748472, 0.181820454731691316338, 0.153785104635716184504,
                                         0.134336222119956792848, 0.10786364350926381636,  0.156084721408851273367};
constexpr double QS_TLO = 150.0, QS_THI = 399.0;
__device__ __forceinline__ double sat_over_t(double T, double T0, double e00, double a, double b, double& rT) {
  const double f = __dadd_rn(T, -T0), d = __dadd_rn(T, T0);
  rT = recip(T);
  const double s = __dmul_rn(f, recip(d));
  const double z = __dmul_rn(s, s), z2 = __dmul_rn(z, z);
  double e = __fma_rn(ATANH_C[8], z2, ATANH_C[6]), o = __fma_rn(ATANH_C[7], z2, ATANH_C[5]);
  e = __fma_rn(e, z2, ATANH_C[4]);
  o = __fma_rn(o, z2, ATANH_C[3]);
  e = __fma_rn(e, z2, ATANH_C[2]);
  o = __fma_rn(o, z2, ATANH_C[1]);
  e = __fma_rn(e, z2, ATANH_C[0]);
  const double l = __fma_rn(__dmul_rn(s, z), __fma_rn(o, z, e), __dadd_rn(s, s));
  const double x = __fma_rn(b, quot(f, T, rT), __dmul_rn(a, l));
  const double ex = exp_reduced(x);
  return __dmul_rn(__dmul_rn(e00, ex), rT);
}
#endif

}  // namespace SHIELD_ARITH
}  // namespace shield
