// The fused GFDL microphysics step: one thread per model level, one group of
// NW warps per column.
//
// Restates Microphysics.__call__ (pySHiELD/stencils/microphysics.py:1981-2263):
// fields_init, ntimes x [warm_rain(first), sedimentation, warm_rain, icloud],
// fields_update, all inside one launch.
//
// Layout of the work:
//  * a block owns G consecutive columns; column g of the block is served by
//    NW = ceil(L / 32) warps, and thread (warp w, lane l) of that group holds
//    level k = 32 w + l (k = 0 is the model top). A warp therefore covers 32
//    adjacent levels, whose physics takes similar branches, and each thread
//    keeps one level's state in registers for the whole step;
//  * the 14 input fields (13 state fields + the persistent cloud-fraction
//    accumulator) are staged once through shared memory with coalesced loads
//    (consecutive threads read consecutive columns of an i-fastest field, or
//    consecutive levels of a k-fastest one); the same tiles carry the outputs
//    back, so HBM traffic is the algorithmic bytes;
//  * vertical operations are warp shuffles plus a carry between the group's
//    warps through shared memory, synchronised by the group's own named
//    barrier: the column any() flags (bar.red.or), the implicit
//    sedimentation, heating and momentum recurrences (first-order linear in
//    the level above, as warp scans of affine maps), the height sweep (a
//    suffix sum) and neighbour reads.
#pragma once

#include "mp_physics.cuh"
#include "mp_physics_mixed.cuh"

namespace shield {
inline namespace SHIELD_ARITH {

#define FULLMASK 0xffffffffu

template <int NW>
struct Tiles {
  static constexpr int RP = 32 * NW + 1;  // doubles per (field, column) row; odd pitch
  static constexpr int SCR = 8 * NW + 8;  // per-column scratch doubles per parity
};

// Vertical operations of one column group. Every thread of the group calls
// the same sequence of operations (group-uniform control flow); each
// operation uses the next of two alternating scratch slots, so one named
// barrier per operation suffices.
template <int NW>
struct Column {
  static constexpr int WP = Tiles<NW>::RP;  // pitch of the work rows
  int w, lane, k, L, bar;
  static constexpr int CV = 10;     // doubles of the column's own values
  static constexpr int NPARK = 13;  // doubles of a thread's slot (ParkSlot, and one to make it odd)
  double* scr;   // 2 * SCR doubles
  double* work;  // 2 * RP doubles, for the sequential vapour borrow: the threads' slots, before they are used
  double* park;  // this thread's slot
  double* cv;    // CV doubles
  int par;

  SHD void sync() const {
    if (NW == 1)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * NW) : "memory");
  }
  // Orders the column's shared accesses before it against those after it,
  // where its operations do not: a one-warp column's are shuffles and votes,
  // which order no memory; every other column's pass a barrier.
  SHD void order() const {
    if constexpr (NW == 1) __syncwarp();
  }
  SHD double* slot() {
    double* s = scr + par * Tiles<NW>::SCR;
    par ^= 1;
    return s;
  }
  // value at level k - 1 (undefined at k = 0)
  SHD double prev(double x) {
    double u = __shfl_up_sync(FULLMASK, x, 1);
    if (NW == 1) return u;
    double* s = slot();
    if (lane == 31) s[w] = x;
    sync();
    if (lane == 0 && w > 0) u = s[w - 1];
    return u;
  }
  SHD bool any(bool p) {
    if (NW == 1) return __any_sync(FULLMASK, p);
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred q, %2, %3, q;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)p), "r"(bar), "r"(32 * NW)
        : "memory");
    return r != 0;
  }
  // any() over every thread that shares this object's barrier: the whole
  // column here (control flow around vertical operations must be uniform
  // over the barrier's threads)
  SHD bool group_any(bool p) { return any(p); }
  // the column's any(p), the barrier group's, and x at level k - 1, from one
  // exchange
  SHD void any_prev(bool p, double x, bool& r, bool& g, double& px) {
    const bool m = __any_sync(FULLMASK, p);
    px = __shfl_up_sync(FULLMASK, x, 1);
    r = m;
    if (NW > 1) {
      double* s = slot();
      unsigned* su = reinterpret_cast<unsigned*>(s + NW);
      if (lane == 31) {
        s[w] = x;
        su[w] = m ? 1u : 0u;
      }
      sync();
      if (lane == 0 && w > 0) px = s[w - 1];
      unsigned o = 0;
#pragma unroll
      for (int u = 0; u < NW; ++u) o |= su[u];
      r = o != 0;
    }
    g = r;
  }
  // the first level where p holds (1 << 30: none) and x at level k - 1, from
  // one exchange
  template <int N>
  SHD int first_prevN(bool p, const double (&x)[N], double (&px)[N]) {
    const unsigned m = __ballot_sync(FULLMASK, p);
    const int mine = m ? 32 * w + __ffs(m) - 1 : 1 << 30;
#pragma unroll
    for (int n = 0; n < N; ++n) px[n] = __shfl_up_sync(FULLMASK, x[n], 1);
    if (NW == 1) return mine;
    double* s = slot();
    int* si = reinterpret_cast<int*>(s + N * NW);
    if (lane == 31) {
#pragma unroll
      for (int n = 0; n < N; ++n) s[N * w + n] = x[n];
      si[w] = mine;
    }
    sync();
    if (lane == 0 && w > 0) {
#pragma unroll
      for (int n = 0; n < N; ++n) px[n] = s[N * (w - 1) + n];
    }
    int f = si[0];
#pragma unroll
    for (int u = 1; u < NW; ++u) f = min(f, si[u]);
    return f;
  }
  // N top-down affine scans (scanN), their values at level k - 1, and the
  // column's any() of N flags, from one exchange
  template <int N>
  SHD void scanN_prev_any(const double (&a)[N], const double (&b)[N], bool (&p)[N], double (&x)[N], double (&xp)[N]) {
    double A[N], B[N];
    unsigned m = 0;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      A[n] = a[n];
      B[n] = b[n];
      m |= (__any_sync(FULLMASK, p[n]) ? 1u : 0u) << n;
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const double pA = __shfl_up_sync(FULLMASK, A[n], d);
        const double pB = __shfl_up_sync(FULLMASK, B[n], d);
        if (lane >= d) {
          A[n] = A[n] + B[n] * pA;
          B[n] = B[n] * pB;
        }
      }
    }
    if (NW > 1) {
      double* s = slot();
      unsigned* su = reinterpret_cast<unsigned*>(s + 2 * N * NW);
      if (lane == 31) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
          s[2 * N * w + 2 * n] = A[n];
          s[2 * N * w + 2 * n + 1] = B[n];
        }
        su[w] = m;
      }
      sync();
#pragma unroll
      for (int n = 0; n < N; ++n) {
        double X = 0.0;
        for (int u = 0; u < w; ++u) X = s[2 * N * u + 2 * n] + s[2 * N * u + 2 * n + 1] * X;
        x[n] = A[n] + B[n] * X;
        xp[n] = X;
      }
      m = su[0];
#pragma unroll
      for (int u = 1; u < NW; ++u) m |= su[u];
    } else {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        x[n] = A[n];
        xp[n] = 0.0;
      }
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const double v = __shfl_up_sync(FULLMASK, x[n], 1);
      if (lane > 0) xp[n] = v;
      p[n] = (m >> n) & 1u;
    }
  }
  SHD int min_int(int v) {
    v = __reduce_min_sync(FULLMASK, v);
    if (NW == 1) return v;
    double* s = slot();
    int* si = reinterpret_cast<int*>(s);
    if (lane == 0) si[w] = v;
    sync();
    int m = si[0];
#pragma unroll
    for (int u = 1; u < NW; ++u) m = min(m, si[u]);
    return m;
  }
  // values of x and y at level k0 (every level receives them)
  SHD void bcast2(double x, double y, int k0, double& x0, double& y0) {
    const int w0 = k0 >> 5, l0 = k0 & 31;
    x0 = __shfl_sync(FULLMASK, x, l0);
    y0 = __shfl_sync(FULLMASK, y, l0);
    if (NW == 1) return;
    double* s = slot();
    if (w == w0 && lane == 0) {
      s[0] = x0;
      s[1] = y0;
    }
    sync();
    x0 = s[0];
    y0 = s[1];
  }
  // X_k = a_k + b_k X_{k-1} from the top down (b must vanish at k = 0)
  SHD double scan_affine(double a, double b) {
    double A = a, B = b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      double pA = __shfl_up_sync(FULLMASK, A, d);
      double pB = __shfl_up_sync(FULLMASK, B, d);
      if (lane >= d) {
        A = A + B * pA;
        B = B * pB;
      }
    }
    if (NW == 1) return A;
    double* s = slot();
    if (lane == 31) {
      s[2 * w] = A;
      s[2 * w + 1] = B;
    }
    sync();
    double X = 0.0;
    for (int u = 0; u < w; ++u) X = s[2 * u] + s[2 * u + 1] * X;
    return A + B * X;
  }
  // two independent scans sharing one barrier
  SHD void scan_affine2(double a1, double b1, double a2, double b2, double& x1, double& x2) {
    double A1 = a1, B1 = b1, A2 = a2, B2 = b2;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      double pA1 = __shfl_up_sync(FULLMASK, A1, d), pB1 = __shfl_up_sync(FULLMASK, B1, d);
      double pA2 = __shfl_up_sync(FULLMASK, A2, d), pB2 = __shfl_up_sync(FULLMASK, B2, d);
      if (lane >= d) {
        A1 = A1 + B1 * pA1;
        B1 = B1 * pB1;
        A2 = A2 + B2 * pA2;
        B2 = B2 * pB2;
      }
    }
    if (NW == 1) {
      x1 = A1;
      x2 = A2;
      return;
    }
    double* s = slot();
    if (lane == 31) {
      s[4 * w] = A1;
      s[4 * w + 1] = B1;
      s[4 * w + 2] = A2;
      s[4 * w + 3] = B2;
    }
    sync();
    double X1 = 0.0, X2 = 0.0;
    for (int u = 0; u < w; ++u) {
      X1 = s[4 * u] + s[4 * u + 1] * X1;
      X2 = s[4 * u + 2] + s[4 * u + 3] * X2;
    }
    x1 = A1 + B1 * X1;
    x2 = A2 + B2 * X2;
  }
  // values at levels k - 1 of N fields with one barrier (undefined at k = 0)
  template <int N>
  SHD void prevN(const double (&x)[N], double (&px)[N]) {
#pragma unroll
    for (int n = 0; n < N; ++n) px[n] = __shfl_up_sync(FULLMASK, x[n], 1);
    if (NW == 1) return;
    double* s = slot();
    if (lane == 31) {
#pragma unroll
      for (int n = 0; n < N; ++n) s[N * w + n] = x[n];
    }
    sync();
    if (lane == 0 && w > 0) {
#pragma unroll
      for (int n = 0; n < N; ++n) px[n] = s[N * (w - 1) + n];
    }
  }
  // values at levels k - 1 and k + 1 of N fields with one barrier
  template <int N>
  SHD void nbrsN(const double (&x)[N], double (&xp)[N], double (&xn)[N]) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      xp[n] = __shfl_up_sync(FULLMASK, x[n], 1);
      xn[n] = __shfl_down_sync(FULLMASK, x[n], 1);
    }
    if (NW == 1) return;
    double* s = slot();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (lane == 0) s[2 * (N * w + n)] = x[n];
      if (lane == 31) s[2 * (N * w + n) + 1] = x[n];
    }
    sync();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (lane == 0 && w > 0) xp[n] = s[2 * (N * (w - 1) + n) + 1];
      if (lane == 31 && w < NW - 1) xn[n] = s[2 * (N * (w + 1) + n)];
    }
  }
  // three column any() flags with one barrier
  SHD void any3(bool a, bool b, bool c, bool& ra, bool& rb, bool& rc) {
    const unsigned m = (__any_sync(FULLMASK, a) ? 1u : 0u) | (__any_sync(FULLMASK, b) ? 2u : 0u) |
                       (__any_sync(FULLMASK, c) ? 4u : 0u);
    unsigned r = m;
    if (NW > 1) {
      double* s = slot();
      unsigned* su = reinterpret_cast<unsigned*>(s);
      if (lane == 0) su[w] = m;
      sync();
      r = 0;
#pragma unroll
      for (int u = 0; u < NW; ++u) r |= su[u];
    }
    ra = (r & 1u) != 0;
    rb = (r & 2u) != 0;
    rc = (r & 4u) != 0;
  }
  // N independent top-down affine scans with one barrier
  template <int N>
  SHD void scanN(const double (&a)[N], const double (&b)[N], double (&x)[N]) {
    double A[N], B[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      A[n] = a[n];
      B[n] = b[n];
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const double pA = __shfl_up_sync(FULLMASK, A[n], d);
        const double pB = __shfl_up_sync(FULLMASK, B[n], d);
        if (lane >= d) {
          A[n] = A[n] + B[n] * pA;
          B[n] = B[n] * pB;
        }
      }
    }
    if (NW == 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) x[n] = A[n];
      return;
    }
    double* s = slot();
    if (lane == 31) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        s[2 * N * w + 2 * n] = A[n];
        s[2 * N * w + 2 * n + 1] = B[n];
      }
    }
    sync();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      double X = 0.0;
      for (int u = 0; u < w; ++u) X = s[2 * N * u + 2 * n] + s[2 * N * u + 2 * n + 1] * X;
      x[n] = A[n] + B[n] * X;
    }
  }
  // layer thickness from the BACKWARD height sweep with one barrier:
  // ze_k = zs + sum_{j >= k} (-dz1_j); dz_k = ze_k - ze_{k+1}, dz_{L-1} = ze_{L-1} - zs
  SHD double heights(double t, double zs) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      double v = __shfl_down_sync(FULLMASK, t, d);
      if (lane + d < 32) t = t + v;
    }
    double zn_in_warp = __shfl_down_sync(FULLMASK, t, 1);  // suffix at k + 1 within the warp
    double c = 0.0, cn = 0.0;
    if (NW > 1) {
      double* s = slot();
      if (lane == 0) s[w] = t;
      sync();
      for (int u = NW - 1; u > w; --u) c = c + s[u];
      // for lane 31 the level below is lane 0 of warp w + 1: its suffix is
      // s[w + 1] plus the carry from the warps below it
      if (lane == 31 && w < NW - 1) {
        for (int u = NW - 1; u > w + 1; --u) cn = cn + s[u];
        zn_in_warp = s[w + 1];
      }
    }
    const double ze = zs + (t + c);
    double zn;
    if (lane == 31)
      zn = zs + (zn_in_warp + cn);
    else
      zn = zs + (zn_in_warp + c);
    return (k == L - 1) ? ze - zs : ze - zn;
  }
  // ---------------------------------------------- exchanges of the adjoint
  // values at level k + 1 of N fields with one barrier (undefined at the
  // last level of the group)
  template <int N>
  SHD void nextN(const double (&x)[N], double (&xn)[N]) {
#pragma unroll
    for (int n = 0; n < N; ++n) xn[n] = __shfl_down_sync(FULLMASK, x[n], 1);
    if (NW == 1) return;
    double* s = slot();
    if (lane == 0) {
#pragma unroll
      for (int n = 0; n < N; ++n) s[N * w + n] = x[n];
    }
    sync();
    if (lane == 31 && w < NW - 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) xn[n] = s[N * (w + 1) + n];
    }
  }
  // N independent bottom-up affine scans X_k = a_k + c_k X_{k+1} with one
  // barrier (c must vanish at the last level); the adjoints of the
  // top-down recurrences
  template <int N>
  SHD void scanN_rev(const double (&a)[N], const double (&c)[N], double (&x)[N]) {
    double A[N], B[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      A[n] = a[n];
      B[n] = c[n];
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const double pA = __shfl_down_sync(FULLMASK, A[n], d);
        const double pB = __shfl_down_sync(FULLMASK, B[n], d);
        if (lane + d < 32) {
          A[n] = A[n] + B[n] * pA;
          B[n] = B[n] * pB;
        }
      }
    }
    if (NW == 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) x[n] = A[n];
      return;
    }
    double* s = slot();
    if (lane == 0) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        s[2 * N * w + 2 * n] = A[n];
        s[2 * N * w + 2 * n + 1] = B[n];
      }
    }
    sync();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      double X = 0.0;
      for (int u = NW - 1; u > w; --u) X = s[2 * N * u + 2 * n] + s[2 * N * u + 2 * n + 1] * X;
      x[n] = A[n] + B[n] * X;
    }
  }
  SHD double scan_affine_rev(double a, double c) {
    const double aa[1] = {a}, cc[1] = {c};
    double xx[1];
    scanN_rev<1>(aa, cc, xx);
    return xx[0];
  }
  // sum over the column's levels (every level receives it), in a fixed order
  SHD double colsum(double x) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) x = x + __shfl_xor_sync(FULLMASK, x, d);
    if (NW == 1) return x;
    double* s = slot();
    if (lane == 0) s[w] = x;
    sync();
    double t = s[0];
    for (int u = 1; u < NW; ++u) t = t + s[u];
    return t;
  }
};

// P columns of L levels packed one after another on the 32 NWG threads of
// a group, which share one named barrier: thread t of the group holds level
// k = t - c L of column c = t / L; the threads from P L on form an idle tail
// (column slot P). With L = 79, two columns fill 5 warps (158 of 160
// threads) where one column per 3 warps leaves 17 of 96 threads idle.
//
// Every vertical operation is segmented by column: a value never enters
// arithmetic with another column's (the warp scans combine lanes of one
// column only, the carries between warps come from that column's warps, the
// any/first reductions and broadcasts keep a slot per column). A column
// spans SPAN = 3 warps, whole ones except at its ends, so a warp holds parts
// of at most two segments: the one holding its lane 0 (head) and the one
// holding its lane 31 (tail). Control flow around a vertical operation must
// be uniform over the whole group (the group's any()), not only over a
// column. The idle tail reads the last column's slots; its values reach
// nothing.
template <int NWG, int P>
struct PackedColumn {
  static constexpr int T = 32 * NWG;   // threads of the group
  static constexpr int LMAX = T / P;   // longest column that fits
  static constexpr int WP = LMAX + 1;  // pitch of the work rows
  static constexpr int SCR = 8 * NWG + 8 + 4 * (P + 1);  // scratch doubles per parity
  static constexpr int SPAN = 3;
  static_assert(P == 2 && LMAX == 80, "a column of 65..80 levels, two to a group: SPAN warps each");
  int t, c, k, L, bar;
  int wf;      // first warp of this thread's column
  int off;     // 1: the column starts inside that warp
  static constexpr int CV = 10;     // doubles of a column's own values
  static constexpr int NPARK = 13;  // doubles of a thread's slot (ParkSlot, and one to make it odd)
  static_assert((P + 1) * 2 * WP <= T * NPARK, "the work rows lie in the threads' slots");
  double* scr;   // 2 * SCR doubles
  double* work;  // this column's two work rows (WP doubles each), in the threads' slots before they are used
  double* park;  // this thread's slot
  double* cv;    // the column's CV doubles
  int par;

  // scr_grp / work_grp: the group's scratch, and its threads' slots with its P + 1 columns' values
  SHD void init(int t_, int L_, int bar_, double* scr_grp, double* work_grp) {
    t = t_;
    L = L_;
    bar = bar_;
    c = t / L;
    if (c > P) c = P;
    k = t - c * L;
    const int s0 = min(c, P - 1) * L;
    wf = s0 >> 5;
    off = (s0 & 31) != 0;
    scr = scr_grp;
    work = work_grp + (size_t)c * 2 * WP;
    park = work_grp + (size_t)t * NPARK;
    cv = work_grp + (size_t)T * NPARK + c * CV;
    par = 0;
  }
  SHD int w() const { return t >> 5; }
  SHD int lane() const { return t & 31; }
  // levels of this thread's column above it in its warp
  SHD int above() const { return min(lane(), k); }
  // lanes of this warp in this column (k <= lane: the column starts here)
  SHD unsigned segmask() const {
    const unsigned from = k <= lane() ? FULLMASK << (lane() - k) : FULLMASK;
    const int last = lane() + (c < P ? L - 1 - k : T);  // lane of its last level
    return last < 31 ? from & ((2u << last) - 1u) : from;
  }

  SHD void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(T) : "memory"); }
  SHD void order() const {}  // its operations pass the group's barrier
  SHD double* slot() {
    double* s = scr + par * SCR;
    par ^= 1;
    return s;
  }
  // OR of this column's per-warp words: a pair per warp, of the segment
  // holding its lane 0 and the one holding its lane 31
  SHD void put_part(unsigned* s, unsigned bits) const {
    if (lane() == 0) s[2 * w()] = bits;
    if (lane() == 31) s[2 * w() + 1] = bits;
  }
  SHD unsigned or_parts(const unsigned* s) const {
    unsigned r = s[2 * wf + off];
#pragma unroll
    for (int j = 1; j < SPAN; ++j) r |= s[2 * (wf + j)];
    return r;
  }
  SHD bool group_any(bool p) {
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred q, %2, %3, q;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)p), "r"(bar), "r"(T)
        : "memory");
    return r != 0;
  }
  // ------------------------------------------------ neighbour exchanges
  // (values of another column, read at a column's ends, are not used by
  // the callers, which select the boundary value at k = 0 / k = L - 1)
  template <int N>
  SHD void nbrsN(const double (&x)[N], double (&xp)[N], double (&xn)[N]) {
    double* s = slot();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      xp[n] = __shfl_up_sync(FULLMASK, x[n], 1);
      xn[n] = __shfl_down_sync(FULLMASK, x[n], 1);
      if (lane() == 0) s[2 * (N * w() + n)] = x[n];
      if (lane() == 31) s[2 * (N * w() + n) + 1] = x[n];
    }
    sync();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (lane() == 0 && w() > 0) xp[n] = s[2 * (N * (w() - 1) + n) + 1];
      if (lane() == 31 && w() < NWG - 1) xn[n] = s[2 * (N * (w() + 1) + n)];
    }
  }
  // the column's any(p), the group's, and x at level k - 1, from one exchange
  SHD void any_prev(bool p, double x, bool& r, bool& g, double& px) {
    const unsigned m = __ballot_sync(FULLMASK, p);
    px = __shfl_up_sync(FULLMASK, x, 1);
    double* s = slot();
    unsigned* su = reinterpret_cast<unsigned*>(s + NWG);
    put_part(su, (m & segmask()) ? 1u : 0u);
    if (lane() == 31) s[w()] = x;
    sync();
    if (lane() == 0 && w() > 0) px = s[w() - 1];
    r = or_parts(su) != 0;
    unsigned o = 0;
#pragma unroll
    for (int u = 0; u < 2 * NWG; ++u) o |= su[u];
    g = o != 0;
  }
  // the first level of the column where p holds (1 << 30: none) and x at
  // level k - 1, from one exchange
  template <int N>
  SHD int first_prevN(bool p, const double (&x)[N], double (&px)[N]) {
    const unsigned m = __ballot_sync(FULLMASK, p) & segmask();
#pragma unroll
    for (int n = 0; n < N; ++n) px[n] = __shfl_up_sync(FULLMASK, x[n], 1);
    double* s = slot();
    unsigned* su = reinterpret_cast<unsigned*>(s + N * NWG);
    // 127 less the level, so that the first level is the largest value
    const unsigned v = m ? 128u - (unsigned)(k - lane() + __ffs(m)) : 0u;
    put_part(su, v);
    if (lane() == 31) {
#pragma unroll
      for (int n = 0; n < N; ++n) s[N * w() + n] = x[n];
    }
    sync();
    if (lane() == 0 && w() > 0) {
#pragma unroll
      for (int n = 0; n < N; ++n) px[n] = s[N * (w() - 1) + n];
    }
    unsigned f = su[2 * wf + off];
#pragma unroll
    for (int j = 1; j < SPAN; ++j) f = max(f, su[2 * (wf + j)]);
    return f ? 127 - (int)f : 1 << 30;
  }
  // values of N fields at level k0 of this column
  template <int N>
  SHD void bcastN(const double (&x)[N], int k0, double (&x0)[N]) {
    double* s = slot();
    if (k == k0 && c < P) {
#pragma unroll
      for (int n = 0; n < N; ++n) s[N * c + n] = x[n];
    }
    sync();
    const int cc = c < P ? c : P - 1;
#pragma unroll
    for (int n = 0; n < N; ++n) x0[n] = s[N * cc + n];
  }
  SHD void bcast2(double x, double y, int k0, double& x0, double& y0) {
    const double v[2] = {x, y};
    double r[2];
    bcastN<2>(v, k0, r);
    x0 = r[0];
    y0 = r[1];
  }
  // ------------------------------------------------ recurrences
  // N independent top-down affine scans X_k = a_k + b_k X_{k-1} (b must
  // vanish at k = 0), their values at level k - 1, and the column's any() of
  // N flags, from one exchange
  template <int N>
  SHD void scanN_prev_any(const double (&a)[N], const double (&b)[N], bool (&p)[N], double (&x)[N], double (&xp)[N]) {
    double A[N], B[N];
    unsigned bits = 0;
    const unsigned seg = segmask();
#pragma unroll
    for (int n = 0; n < N; ++n) {
      A[n] = a[n];
      B[n] = b[n];
      bits |= ((__ballot_sync(FULLMASK, p[n]) & seg) != 0u ? 1u : 0u) << n;
    }
    const int up = above();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const double pA = __shfl_up_sync(FULLMASK, A[n], d);
        const double pB = __shfl_up_sync(FULLMASK, B[n], d);
        if (up >= d) {
          A[n] = A[n] + B[n] * pA;
          B[n] = B[n] * pB;
        }
      }
    }
    double* s = slot();
    unsigned* su = reinterpret_cast<unsigned*>(s + 2 * N * NWG);
    put_part(su, bits);
    if (lane() == 31) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        s[2 * N * w() + 2 * n] = A[n];
        s[2 * N * w() + 2 * n + 1] = B[n];
      }
    }
    sync();
    // the carry from this column's earlier warps, at most SPAN - 1 (lane 31 of each is in it)
#pragma unroll
    for (int n = 0; n < N; ++n) {
      double X = 0.0;
#pragma unroll
      for (int j = 0; j < SPAN - 1; ++j)
        if (wf + j < w()) X = s[2 * N * (wf + j) + 2 * n] + s[2 * N * (wf + j) + 2 * n + 1] * X;
      x[n] = (w() > wf) ? A[n] + B[n] * X : A[n];
      const double v = __shfl_up_sync(FULLMASK, x[n], 1);
      xp[n] = lane() > 0 ? v : X;
    }
    bits = or_parts(su);
#pragma unroll
    for (int n = 0; n < N; ++n) p[n] = (bits >> n) & 1u;
  }
  SHD double scan_affine(double a, double b) {
    const double aa[1] = {a}, bb[1] = {b};
    double xx[1], xp[1];
    bool p[1] = {false};
    scanN_prev_any<1>(aa, bb, p, xx, xp);
    return xx[0];
  }
  SHD void scan_affine2(double a1, double b1, double a2, double b2, double& x1, double& x2) {
    const double aa[2] = {a1, a2}, bb[2] = {b1, b2};
    double xx[2], xp[2];
    bool p[2] = {false, false};
    scanN_prev_any<2>(aa, bb, p, xx, xp);
    x1 = xx[0];
    x2 = xx[1];
  }
  // layer thickness from the BACKWARD height sweep:
  // ze_k = zs + sum_{j >= k} (-dz1_j); dz_k = ze_k - ze_{k+1}, dz_{L-1} = ze_{L-1} - zs
  SHD double heights(double x, double zs) {
    const int below = min(31 - lane(), (c < P ? L : T - P * L) - 1 - k);  // levels of the column below in the warp
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double v = __shfl_down_sync(FULLMASK, x, d);
      if (below >= d) x = x + v;
    }
    double zn_in_warp = __shfl_down_sync(FULLMASK, x, 1);  // suffix at k + 1 within the warp
    double* s = slot();
    // lane 0 of each of this column's later warps holds that warp's part
    if (lane() == 0) s[w()] = x;
    sync();
    const int wl = wf + SPAN - 1;
    double cc = 0.0, cn = 0.0;
#pragma unroll
    for (int j = 0; j < SPAN - 1; ++j)
      if (wl - j > w()) cc = cc + s[wl - j];
    if (lane() == 31 && w() < wl) {
#pragma unroll
      for (int j = 0; j < SPAN - 2; ++j)
        if (wl - j > w() + 1) cn = cn + s[wl - j];
      zn_in_warp = s[w() + 1];
    }
    const double ze = zs + (x + cc);
    const double zn = (lane() == 31) ? zs + (zn_in_warp + cn) : zs + (zn_in_warp + cc);
    return (k == L - 1) ? ze - zs : ze - zn;
  }
};

// Implicit upwind fall of one species (use_ppm = False): q is the dry mixing
// ratio (updated), dtf the fall time step; returns the cumulative mass flux
// m1 at this level (microphysics.py:454-507 and the ice/snow/graupel repeats).
//
// The reference accumulates m1_k = (m1_{k-1} + q_k) - qm_k level by level.
// With r_k the density from the implicit recurrence, r_k (dz_k + dd_k) =
// q_k + dd_{k-1} r_{k-1}, that running sum telescopes to m1_k = dd_k r_k:
// the mass leaving the bottom of level k. The telescoped form is used here.
// It equals the running sum in exact arithmetic, but it does not cancel: the
// running sum loses all its digits when little mass reaches the ground.
//
// vtp: the fall speed at the level above; fp: the flux there (the same
// product that level forms).
template <class Col>
SHD double implicit_fall(Col& C, double& q, double vt, double vtp, double dz, double dp1, bool valid, double dtf,
                         double& fp) {
  const double dd = dtf * vt, ddp = dtf * vtp;
  const double qmass = valid ? q * dp1 : 0.0;
  const Divisor<double> by_D(dz + dd);
  double a[1] = {by_D(qmass)}, b[1] = {(C.k == 0) ? 0.0 : by_D(ddp)};
  if (!valid) {
    a[0] = 0.0;
    b[0] = 0.0;
  }
  double r[1], rp[1];
  bool p[1] = {false};
  C.template scanN_prev_any<1>(a, b, p, r, rp);
  fp = valid ? ddp * rp[0] : 0.0;
  if (valid) q = qdiv(r[0] * dz, dp1);
  return valid ? dd * r[0] : 0.0;
}

// Implicit heating by falling condensate (microphysics.py:516-557 with
// C_LIQ, :1176-1217 with C_ICE); fp is the flux at the level above.
template <class Col>
SHD void sedi_heat(Col& C, const MpConst& K, double& tz, double dz1, double dp1, double qv, double ql,
                   double qr, double qi, double qs, double qg, double flux, double fp, bool valid, double c_cond) {
  const double dgz = -0.5 * K.GRAV * dz1;
  const double cvn = dp1 * (K.CV_AIR + qv * K.CV_VAP + (qr + ql) * K.C_LIQ + (qi + qs + qg) * K.C_ICE);
  double a, b;
  if (C.k == 0) {
    const double tmp = cvn + flux * c_cond;
    a = tz + qdiv(flux * dgz, tmp);
    b = 0.0;
  } else {
    const Divisor<double> by_D(cvn + c_cond * flux);
    a = by_D((cvn + c_cond * (flux - fp)) * tz + dgz * (fp + flux));
    b = by_D(fp * c_cond);
  }
  if (!valid) {
    a = tz;
    b = 0.0;
  }
  tz = C.scan_affine(a, b);
}

// Vertical-velocity update by one falling species given the flux and fall
// speed at this level and the level above (microphysics.py:492-515).
SHD double w_update(int k, double w, double dm, double flux, double vt, double fp, double vp) {
  if (k == 0) return qdiv(dm * w + flux * vt, dm - flux);
  return qdiv(dm * w - fp * vp + flux * vt, dm + fp - flux);
}

// Monotone vertical slope for autoconversion (microphysics.py:595-620,
// 1341-1367), before the h_var floor: dq_k = 0.5 (q_k - q_{k-1}).
template <class Col>
SHD double mono_slope(Col& C, double q) {
  const double x[1] = {q};
  double xp[1], xn[1];
  C.template nbrsN<1>(x, xp, xn);
  const double dq = 0.5 * (q - xp[0]);
  const double dqn = 0.5 * (xn[0] - q);
  double v = 0.0;
  if (C.k >= 1 && C.k <= C.L - 2) {
    v = 0.5 * qmin(fabs(dq + dqn), 0.5 * q);
    if (dq * dqn <= 0.0) {
      if (dq > 0.0)
        v = qmin(v, qmin(dq, -dqn));
      else
        v = 0.0;
    }
  }
  return v;
}

// ----------------------------------------------------------------- layouts
// How a block's threads map onto its G columns. A layout gives the column
// type the stages run on, the block's thread count, the pitch RP (>= L) of
// the staging tiles, and the scratch and work doubles of each of its NGRP
// barrier groups.
//
// ColumnLayout<NW, G>: each of the G columns on NW whole warps of its own
// (level k = 32 w + lane); one barrier group per column.
template <int NW, int G_>
struct ColumnLayout {
  using Col = Column<NW>;
  static constexpr int G = G_;
  static constexpr int NGRP = G_;
  static_assert(NW == 1 || G_ <= 15, "barrier ids are 1 + g, of 16 (0 is the block's); a one-warp column uses none");
  static constexpr int THREADS = 32 * NW * G_;
  static constexpr int RP = Tiles<NW>::RP;
  static constexpr int SCR = Tiles<NW>::SCR;
  static constexpr int WORK = THREADS / G_ * Col::NPARK + Col::CV;
  // set up thread tid's column object; returns its block column (G: none)
  static SHD int setup(Col& C, int tid, int L, double* scr, double* work) {
    const int g = tid / (32 * NW);
    C.w = (tid >> 5) % NW;
    C.lane = tid & 31;
    C.k = 32 * C.w + C.lane;
    C.L = L;
    C.bar = 1 + g;
    C.scr = scr + (size_t)g * 2 * SCR;
    C.work = work + (size_t)g * WORK;
    C.park = C.work + (tid % (32 * NW)) * Col::NPARK;
    C.cv = C.work + 32 * NW * Col::NPARK;
    C.par = 0;
    return g;
  }
};

// PackedLayout<NWG, P, NGRP>: NGRP groups of NWG warps, each holding P
// columns back to back (PackedColumn); G = P NGRP columns per block.
template <int NWG, int P, int NGRP_>
struct PackedLayout {
  using Col = PackedColumn<NWG, P>;
  static constexpr int G = P * NGRP_;
  static constexpr int NGRP = NGRP_;
  static constexpr int THREADS = 32 * NWG * NGRP_;
  static constexpr int RP = Col::WP;
  static constexpr int SCR = Col::SCR;
  static constexpr int WORK = 32 * NWG * Col::NPARK + (P + 1) * Col::CV;
  static SHD int setup(Col& C, int tid, int L, double* scr, double* work) {
    const int gi = tid / (32 * NWG);
    C.init(tid % (32 * NWG), L, 1 + gi, scr + (size_t)gi * 2 * SCR, work + (size_t)gi * WORK);
    return C.c < P ? gi * P + C.c : G;
  }
};

// ----------------------------------------------------------------- staging
// Shared memory: N_IN tiles of G rows of RP doubles (field f, block column g,
// level k at (f * G + g) * RP + k), then the groups' scratch (NGRP x 2 x SCR
// doubles), then their work rows for the rare sequential vapour borrow.
template <class LY>
struct Smem {
  static constexpr size_t tiles = (size_t)N_IN * LY::G * LY::RP;
  static constexpr size_t scratch = tiles;
  static constexpr size_t work = scratch + (size_t)LY::NGRP * 2 * LY::SCR;
  static constexpr size_t total = work + (size_t)LY::NGRP * LY::WORK;
  static constexpr size_t bytes = total * sizeof(double);
};

// Element e < G L of a field's block tile for thread e, in the two memory
// orders: i-fastest storages take consecutive columns on consecutive
// threads (g = e % G, k = e / G), k-fastest ones consecutive levels
// (g = e / L, k = e % L). Every layout has at least G L threads, so each
// thread moves at most one element of each field, and all loads of a stage
// are issued before any store: one memory round trip per stage.
SHD int div_nx(const MpArgs& A, int64_t n) { return (int)(((uint64_t)(uint32_t)n * A.by_nx.m) >> A.by_nx.s); }

struct StageMap {
  int g, k, gk, kk;
  bool ok, okk;
  int64_t i, j, ik, jk;
  template <int G>
  SHD void set(const MpArgs& A, int tid, int64_t c0) {
    g = tid % G;
    k = tid / G;
    const int64_t col = c0 + g;
    ok = col < A.ncol && k < A.nz;
    j = ok ? div_nx(A, col) : 0;
    i = ok ? col - j * A.nx : 0;
  }
  // the k-fastest order
  template <int G>
  SHD void set_kfast(const MpArgs& A, int tid, int64_t c0) {
    gk = tid / A.nz;
    kk = tid - gk * A.nz;
    const int64_t colk = c0 + gk;
    okk = gk < G && colk < A.ncol;
    jk = okk ? div_nx(A, colk) : 0;
    ik = okk ? colk - jk * A.nx : 0;
  }
};

// With one set of strides in every field of the caller (same_strides: NDSL
// storages of one shape), the staging forms one offset; otherwise each
// field its own, in its own memory order. The general form's 64-bit column
// divisions and 26 address computations were 1,250 of the step's 8,600
// instructions per warp.
template <class LY>
SHD void stage_in(const MpArgs& A, double* sm, int64_t c0) {
  constexpr int RP = LY::RP, G = LY::G;
  StageMap M;
  M.template set<G>(A, threadIdx.x, c0);
  double v[N_IN];
  if (A.same_strides) {
    const Fld3& F = A.in[0];
    const int64_t o = M.i * F.si + M.j * F.sj + (int64_t)M.k * F.sk;
    const int64_t oq = c0 + M.g + M.k * A.ncol;
    if (!M.ok) return;
#pragma unroll
    for (int f = 0; f < IN_QAZ; ++f) v[f] = A.in[f].p[o];
    v[IN_QAZ] = A.in[IN_QAZ].p[oq];
#pragma unroll
    for (int f = 0; f < N_IN; ++f) sm[(f * G + M.g) * RP + M.k] = v[f];
    return;
  }
  M.template set_kfast<G>(A, threadIdx.x, c0);
#pragma unroll
  for (int f = 0; f < N_IN; ++f) {
    const Fld3 F = A.in[f];
    v[f] = 0.0;
    if (F.sk == 1) {
      if (M.okk) v[f] = F.p[M.ik * F.si + M.jk * F.sj + M.kk];
    } else if (M.ok) {
      v[f] = F.p[M.i * F.si + M.j * F.sj + (int64_t)M.k * F.sk];
    }
  }
#pragma unroll
  for (int f = 0; f < N_IN; ++f) {
    const Fld3 F = A.in[f];
    if (F.sk == 1) {
      if (M.okk) sm[(f * G + M.gk) * RP + M.kk] = v[f];
    } else if (M.ok) {
      sm[(f * G + M.g) * RP + M.k] = v[f];
    }
  }
}

enum OutMode { OM_SKIP = 0, OM_ADD = 1, OM_ADD_K1 = 2, OM_SET = 3 };

SHD int out_mode(const MpConst& K, int o) {
  int m = OM_ADD;
  if (o == OUT_UDT || o == OUT_VDT) m = K.sedi_transport ? OM_ADD_K1 : OM_SKIP;
  if (o == OUT_QA_DT && K.do_qa) m = OM_SET;
  if (o == OUT_W) m = K.do_sedi_w ? OM_SET : OM_SKIP;
  if (o == OUT_QAZ) m = OM_SET;
  return m;
}

// tendency of a step that starts from zero tendencies
SHD double fresh_tendency(int mode, bool k1, double v) {
  return (mode == OM_SET) ? v : (mode == OM_ADD || (mode == OM_ADD_K1 && k1)) ? __dadd_rn(0.0, v) : 0.0;
}

template <class LY>
SHD void stage_out(const MpArgs& A, const double* sm, int64_t c0) {
  constexpr int RP = LY::RP, G = LY::G;
  const MpConst& K = A.K;
  StageMap M;
  M.template set<G>(A, threadIdx.x, c0);
  double old[N_OUT];
  if (A.same_strides) {
    const Fld3& F = A.in[0];
    const int64_t o = M.i * F.si + M.j * F.sj + (int64_t)M.k * F.sk;
    const int64_t oq = c0 + M.g + M.k * A.ncol;
    if (!M.ok) return;
    const bool k1 = M.k >= 1;  // the winds' tendencies are written below the top level
    if (A.fresh) {
#pragma unroll
      for (int n = 0; n < OUT_W; ++n)
        A.out[n].p[o] = fresh_tendency(out_mode(K, n), k1, sm[(n * G + M.g) * RP + M.k]);
    } else {
#pragma unroll
      for (int n = 0; n < OUT_W; ++n) {
        const int m = out_mode(K, n);
        old[n] = (m == OM_ADD || (m == OM_ADD_K1 && k1)) ? A.out[n].p[o] : 0.0;
      }
#pragma unroll
      for (int n = 0; n < OUT_W; ++n) {
        const int m = out_mode(K, n);
        const double v = sm[(n * G + M.g) * RP + M.k];
        if (m == OM_SET || m == OM_ADD || (m == OM_ADD_K1 && k1)) A.out[n].p[o] = (m == OM_SET) ? v : old[n] + v;
      }
    }
    if (out_mode(K, OUT_W) == OM_SET) A.out[OUT_W].p[o] = sm[(OUT_W * G + M.g) * RP + M.k];
    A.out[OUT_QAZ].p[oq] = sm[(OUT_QAZ * G + M.g) * RP + M.k];
    return;
  }
  M.template set_kfast<G>(A, threadIdx.x, c0);
  int mode[N_OUT];
  double* dst[N_OUT];
#pragma unroll
  for (int o = 0; o < N_OUT; ++o) {
    int m = out_mode(K, o);
    const Fld3 F = A.out[o];
    const bool kf = F.sk == 1;
    const int lev = kf ? M.kk : M.k;
    const bool fresh = A.fresh && o < OUT_W;
    if (!(kf ? M.okk : M.ok) || (!fresh && m == OM_ADD_K1 && lev < 1)) m = OM_SKIP;
    else if (fresh) m = OM_SET;
    mode[o] = m;
    dst[o] = kf ? F.p + M.ik * F.si + M.jk * F.sj + M.kk : F.p + M.i * F.si + M.j * F.sj + (int64_t)M.k * F.sk;
    old[o] = (m == OM_ADD || m == OM_ADD_K1) ? *dst[o] : 0.0;
  }
#pragma unroll
  for (int o = 0; o < N_OUT; ++o) {
    if (mode[o] == OM_SKIP) continue;
    const bool kf = A.out[o].sk == 1;
    double v = kf ? sm[(o * G + M.gk) * RP + M.kk] : sm[(o * G + M.g) * RP + M.k];
    if (A.fresh && o < OUT_W) v = fresh_tendency(out_mode(K, o), (kf ? M.kk : M.k) >= 1, v);
    *dst[o] = (mode[o] == OM_SET) ? v : old[o] + v;
  }
}

// ------------------------------------------------------------ step stages
// The step body as stages, shared by the forward kernels and the adjoint
// (which replays them). Per level: the prognostic state, and the values set
// by fields_init or at the start of each sub-step that later stages read.
struct LevState {
  double qv, ql, qr, qi, qs, qg, tz, w;
};
// the layer geometry a fall works on (the adjoint's column reverses)
struct StepGeom {
  double dp1, den, denfac, dz1, dz;
};
// What a level keeps between its stages, in shared memory: a slot of N_PARK
// doubles per thread (an odd count, so that consecutive threads' slots hit
// distinct banks), and the column's own values. The step is bound by the
// latency of dependent FP64 work, so resident warps decide its rate (a group
// takes the same time alone on an SM as with three others: 33 against 42 us
// at L79), and registers decide those: the state in use stays in registers,
// these values are read where they are needed.
enum ParkSlot { PK_W, PK_DP1, PK_P1, PK_DZ, PK_DZ1, PK_DENFAC, PK_MP, PK_M1SOL, PK_MPSOL, PK_VTR, PK_VTG, PK_VTS };
struct LevelStore {
  double* pk;  // this thread's slot
  double* cv;  // the column's values: fields_init's, written by level 0 and read after the next exchange (or order())
  double den;  // density (start of each sub-step)
  SHD double& w() const { return pk[PK_W]; }      // vertical velocity
  SHD double& dp1() const { return pk[PK_DP1]; }  // fields_init
  SHD double& p1() const { return pk[PK_P1]; }
  SHD double& dz() const { return pk[PK_DZ]; }    // start of each sub-step
  SHD double& dz1() const { return pk[PK_DZ1]; }
  SHD double& denfac() const { return pk[PK_DENFAC]; }
  // the precipitation flux at the level above, summed over the sub-steps; the
  // solid flux of the last sedimentation, here (kept by a recorder) and there
  SHD double& mp() const { return pk[PK_MP]; }
  SHD double& m1_sol() const { return pk[PK_M1SOL]; }
  SHD double& mp_sol() const { return pk[PK_MPSOL]; }
  // the last fall speeds of rain, graupel and snow
  SHD double& vtr() const { return pk[PK_VTR]; }
  SHD double& vtg() const { return pk[PK_VTG]; }
  SHD double& vts() const { return pk[PK_VTS]; }
  SHD double h_var() const { return cv[0]; }
  SHD double rh_adj() const { return cv[1]; }
  SHD double rh_rain() const { return cv[2]; }
  SHD double ccn() const { return cv[3]; }
  SHD double c_praut() const { return cv[4]; }
};

// the column's surface totals, after fields_init's five values: kept and read
// by the bottom level alone
enum ColumnTotal { CV_RAIN = 5, CV_ICE, CV_SNOW, CV_GRAUPEL };

// fields_init (:27-276) for one level from its input values (defaults on
// the padding levels k >= L, whose values never reach a real level).
template <class Col>
SHD void fields_init(Col& C, const MpConst& K, bool valid, double pt, double qvi, double qli, double qri,
                     double qii, double qsi, double qgi, double delp, double wz, double dz0, double land, double area,
                     LevState& S, LevelStore& P) {
  const int k = C.k, L = C.L;
  P.pk = C.park;
  P.cv = C.cv;
  S.tz = pt;
  const double dp1 = delp * (1.0 - qvi);
  const double omq = qdiv(delp, dp1);
  S.qv = qvi * omq;
  S.ql = qli * omq;
  S.qr = qri * omq;
  S.qi = qii * omq;
  S.qs = qsi * omq;
  S.qg = qgi * omq;
  const double den0 = qdiv(-dp1, K.GRAV * dz0);
  const double p1 = den0 * K.RDGAS * pt;
  double ccn;
  if (K.prog_ccn) {
    ccn = 0.0 * 1.0e6;
  } else {
    ccn = (K.ccn_l * land + K.ccn_o * (1.0 - land)) * 1.0e6;
    if (K.use_ccn) {
      double tzb, p1b;
      C.bcast2(S.tz, p1, L - 1, tzb, p1b);
      ccn = qdiv(ccn * K.RDGAS * tzb, p1b);
    }
  }
  const double c_praut = K.cpaut * xpowp(ccn * RHOR, -1.0 / 3.0);
  const double s_leng = qsqrt(qsqrt(area * 1.0e-10));
  const double t_land = K.dw_land * s_leng;
  const double t_ocean = K.dw_ocean * s_leng;
  const double h_var = qmin(0.2, qmax(0.01, t_land * land + t_ocean * (1.0 - land)));
  const double rh_adj = 1.0 - h_var - K.rh_inc;
  if (k == 0) {
    P.cv[0] = h_var;
    P.cv[1] = rh_adj;
    P.cv[2] = qmax(0.35, rh_adj - K.rh_inr);
    P.cv[3] = ccn;
    P.cv[4] = c_praut;
  }

  if (K.fix_negative) {
    fix_negative_point(K, S.qv, S.ql, S.qr, S.qi, S.qs, S.qg, S.tz);
    // FORWARD borrow of negative vapour from the level above (:244-247):
    // a sequential sweep by one thread over the column, taken only when
    // some level above the bottom is negative (in any column sharing the
    // barrier: the sweep leaves a column without such a level unchanged)
    if (C.group_any(valid && k < L - 1 && S.qv < 0.0)) {
      double* wq = C.work;
      double* wd = wq + Col::WP;
      if (valid) {
        wq[k] = S.qv;
        wd[k] = dp1;
      }
      C.sync();
      if (k == 0) {
        for (int kk = 1; kk < L; ++kk) {
          const double pq = wq[kk - 1];
          if (pq < 0.0) wq[kk] = wq[kk] + pq * wd[kk - 1] / wd[kk];
        }
      }
      C.sync();
      if (valid) S.qv = wq[k];
    }
    if (k < L - 1 && S.qv < 0.0) S.qv = 0.0;
    // bottom layer borrows from the layer above (:253-276): the two levels
    // form the same dq
    const double x[2] = {S.qv, dp1};
    double xp[2], xn[2];
    C.template nbrsN<2>(x, xp, xn);
    if (k == L - 2 || k == L - 1) {
      const bool bot = k == L - 1;
      const double qb = bot ? S.qv : xn[0], db = bot ? dp1 : xn[1];
      const double qb1 = bot ? xp[0] : S.qv, db1 = bot ? xp[1] : dp1;
      if ((qb < 0.0) && (qb1 > 0.0)) {
        const double dq = qdiv(qmin(-qb * db, qb1 * db1), dp1);
        S.qv = bot ? S.qv + dq : S.qv - dq;
      }
    }
  }
  // After every read of the borrow's work rows, which these slots overlie, and
  // before any read of the column's values: the exchange above lies between,
  // and the next one (heights), or the warp's own synchronisation.
  C.order();
  P.w() = wz;
  P.dp1() = dp1;
  P.p1() = p1;
  P.mp() = 0.0;
}

// density, fall factor and layer thickness at the start of a sub-step
// (warm_rain with is_first, :349-380)
template <class Col>
SHD void substep_geometry(Col& C, const MpConst& K, bool valid, double t0, double dz0, const LevState& S,
                          LevelStore& P) {
  const double den0 = qdiv(-P.dp1(), K.GRAV * dz0);
  const double dz1 = qdiv(dz0 * S.tz, t0);
  P.den = qdiv(den0 * dz0, dz1);
  P.dz1() = dz1;
  P.denfac() = qsqrt(qdiv(SFCRHO, P.den));
  P.dz() = C.heights(valid ? -dz1 : 0.0, K.zs);
}

// Recorder of a stage's intermediate states. The forward kernels pass
// NoRec (every call compiles away); the adjoint's replay passes one that
// stores the states the reverse sweeps start from.
struct NoRec {
  static constexpr bool on = false;
  SHD void state(int, const LevState&) const {}
  SHD void value(int, double) const {}
  SHD void flag(bool) const {}
};

// warm_rain (:280-653) after the geometry: rain evaporation and accretion,
// implicit rain fall with the vertical-velocity transport and heating, then
// autoconversion. Returns the rain flux m1_rain at this level (at the bottom
// level: the surface flux) and m1_prev, the flux at the level above.
// A recorder gets the states after the first evaporation (slot 0), after the
// fall (1) and after the second evaporation (2), the liquid slope (value 0)
// and the column's rain-fall decision.
template <bool MIXED, class Col, class Rec = NoRec>
SHD void warm_rain(Col& C, const MpConst& K, const MpConstF& KF, bool valid, LevState& S, const LevelStore& P,
                   double& m1_rain, double& m1_prev, bool* falls = nullptr, const Rec& rec = Rec()) {
  const int k = C.k;
  double &qv = S.qv, &ql = S.ql, &qr = S.qr, &qi = S.qi, &qs = S.qs, &qg = S.qg, &tz = S.tz;
  if constexpr (Rec::on) S.w = P.w();
  const double dt5 = 0.5 * K.dt_rain;
  m1_rain = 0.0;
  m1_prev = 0.0;
  // the fall speed before it is known whether the column's rain falls (it is
  // VR_MIN without a test of more than qr where none does), so that the
  // decision and the speed above come from one exchange
  double vt, vp;
  if constexpr (MIXED)
    vt = rain_fspeed_m(K, qr, P.den);
  else
    vt = rain_fspeed(K, qr, P.den);
  bool fall, gfall;
  C.any_prev(valid && (qr > QRMIN), vt, fall, gfall, vp);
  if (falls) *falls = fall;
  rec.flag(fall);
  const double vtr = fall ? vt : VF_MIN;
  P.vtr() = vtr;
  // The fall's vertical operations run whenever a column sharing the
  // barrier has falling rain; a column without it takes part with no mass
  // (valid false), which leaves its state unchanged and its flux zero.
  if (gfall) {
    const bool vf = valid && fall;
    if (fall) {
      if constexpr (MIXED)
        revap_racc_m(K, KF, dt5, P.h_var(), qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac());
      else
        revap_racc(K, dt5, P.h_var(), qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac());
    }
    rec.state(0, S);
    const double dp1 = P.dp1();
    const double dm = dp1 * (1.0 + qv + ql + qr + qi + qs + qg);
    m1_rain = implicit_fall(C, qr, vtr, vp, P.dz(), dp1, vf, K.dt_rain, m1_prev);
    if (fall && K.do_sedi_w) P.w() = w_update(k, P.w(), dm, m1_rain, vtr, m1_prev, vp);
    if constexpr (Rec::on) S.w = P.w();
    if (K.do_sedi_heat) sedi_heat(C, K, tz, P.dz1(), P.dp1(), qv, ql, qr, qi, qs, qg, m1_rain, m1_prev, vf, K.C_LIQ);
    rec.state(1, S);
    if (fall) {
      if constexpr (MIXED)
        revap_racc_m(K, KF, dt5, P.h_var(), qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac());
      else
        revap_racc(K, dt5, P.h_var(), qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac());
    }
    rec.state(2, S);
  } else {
    rec.state(0, S);
    rec.state(1, S);
    rec.state(2, S);
  }
  if (K.irain_f != 0) {
    if constexpr (MIXED)
      autoconv_no_subgrid_var_m(K, KF, ql, qr, tz, P.den, P.ccn(), P.c_praut());
    else
      autoconv_no_subgrid_var(K, ql, qr, tz, P.den, P.ccn(), P.c_praut());
  } else {
    double dl;
    if (K.z_slope_liq) {
      dl = mono_slope(C, ql);
      rec.value(0, dl);
      dl = qmax(dl, qmax(QVMIN, P.h_var() * ql));
    } else {
      dl = qmax(QVMIN, P.h_var() * ql);
    }
    if constexpr (MIXED)
      autoconv_subgrid_var_m(K, KF, ql, qr, tz, P.den, P.ccn(), P.c_praut(), dl);
    else
      autoconv_subgrid_var(K, ql, qr, tz, P.den, P.ccn(), P.c_praut(), dl);
  }
}

// sedimentation (:657-1217): fall speeds, cloud ice melting, and the
// implicit falls of ice, snow and graupel with their vertical-velocity
// transport and heating. Stores the solid flux at the level above (with a
// recorder, here too); the bottom level adds the surface fluxes to the column's totals. A
// recorder gets the cloud ice fall speed (value 0).
template <bool MIXED, class Col, class Rec = NoRec>
SHD void sedimentation(Col& C, const MpConst& K, const MpConstF& KF, bool valid, LevState& S,
                       const LevelStore& P, unsigned* flags = nullptr, const Rec& rec = Rec()) {
  const int k = C.k, L = C.L;
  double &qv = S.qv, &ql = S.ql, &qr = S.qr, &qi = S.qi, &qs = S.qs, &qg = S.qg, &tz = S.tz;
  const double dp1 = P.dp1(), dz = P.dz();
  double vti, vts, vtg;
  if constexpr (MIXED)
    fall_speed_m(K, KF, qg, qi, qs, tz, P.den, vtg, vti, vts);
  else
    fall_speed(K, qg, qi, qs, tz, P.den, vtg, vti, vts);
  rec.value(0, vti);
  P.vtg() = vtg;
  P.vts() = vts;
  double m1_sol = 0.0, m1_prev = 0.0;
  // cloud ice melting at and below the first level warmer than tice (:702-746);
  // the fall speeds above come with the same exchange
  const double vt[3] = {vti, vts, vtg};
  double vp[3];
  const int first = C.template first_prevN<3>(valid && tz > K.tice, vt, vp);
  if ((k >= first || k == L - 1) && valid) sedi_ice_melt(K, qv, ql, qr, qi, qs, qg, tz);
  // ice (:773-900), snow (:902-1035) and graupel (:1037-1168): their
  // implicit falls are independent of one another, so the three share one
  // exchange, which also decides which of them fall (in nearly every column
  // of weather some does; a column where none does scans zeros); the
  // vertical-velocity updates, which the reference applies species after
  // species, stay in that order.
  bool f[3] = {valid && (qi > QRMIN), valid && (qs > QRMIN), valid && (qg > QRMIN)};
  double dd[3], ddp[3];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    dd[n] = K.dts * vt[n];
    ddp[n] = K.dts * vp[n];
  }
  const double qq[3] = {qi, qs, qg};
  double ra[3], rb[3], r[3], rp[3];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    const double qmass = valid ? qq[n] * dp1 : 0.0;
    const Divisor<double> by_D(dz + dd[n]);
    ra[n] = by_D(qmass);
    rb[n] = (k == 0) ? 0.0 : by_D(ddp[n]);
    if (!valid) {
      ra[n] = 0.0;
      rb[n] = 0.0;
    }
  }
  C.template scanN_prev_any<3>(ra, rb, f, r, rp);
  const bool fi = f[0] && (K.vi_fac >= 1.0e-5), fs = f[1], fg = f[2];
  if (flags)
    *flags |= (fi ? FLAG_ICE_FALLS : 0u) | (fs ? FLAG_SNOW_FALLS : 0u) | (fg ? FLAG_GRAUPEL_FALLS : 0u) |
              ((unsigned)min(first, L - 1) << FLAG_MELT_SHIFT);
  double flux[3], fp[3];  // of each species, here and at the level above
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    flux[n] = valid ? dd[n] * r[n] : 0.0;
    fp[n] = valid ? ddp[n] * rp[n] : 0.0;
  }
  const Divisor<double> by_dp1(dp1);
  const double dm_i = dp1 * (1.0 + qv + ql + qr + qi + qs + qg);
  if (fi && valid) qi = by_dp1(r[0] * dz);
  const double dm_s = dp1 * (1.0 + qv + ql + qr + qi + qs + qg);
  if (fs && valid) qs = by_dp1(r[1] * dz);
  const double dm_g = dp1 * (1.0 + qv + ql + qr + qi + qs + qg);
  if (fg && valid) qg = by_dp1(r[2] * dz);
  const bool bottom = k == L - 1;
  double w = P.w();
  if (fi) {
    m1_sol = flux[0];
    m1_prev = fp[0];
    if (K.do_sedi_w) w = w_update(k, w, dm_i, flux[0], vti, fp[0], vp[0]);
    if (bottom) C.cv[CV_ICE] += flux[0];
  }
  if (fs) {
    m1_sol = m1_sol + flux[1];
    m1_prev = m1_prev + fp[1];
    if (K.do_sedi_w) w = w_update(k, w, dm_s, flux[1], vts, fp[1], vp[1]);
    if (bottom) C.cv[CV_SNOW] += flux[1];
  }
  if (fg) {
    m1_sol = m1_sol + flux[2];
    m1_prev = m1_prev + fp[2];
    if (K.do_sedi_w) w = w_update(k, w, dm_g, flux[2], vtg, fp[2], vp[2]);
    if (bottom) C.cv[CV_GRAUPEL] += flux[2];
  }
  P.w() = w;
  if constexpr (Rec::on) P.m1_sol() = m1_sol;
  P.mp_sol() = m1_prev;
  if constexpr (Rec::on) S.w = w;
  if (K.do_sedi_heat) sedi_heat(C, K, tz, P.dz1(), dp1, qv, ql, qr, qi, qs, qg, m1_sol, m1_prev, valid, K.C_ICE);
}

// icloud (:1220-1449): instant melting or freezing, the ice slope, the ice
// processes and the saturation adjustment. A recorder gets the state between
// the ice processes and the adjustment (slot 0), the ice slope (value 0) and
// the cloud ice after melting and freezing (value 1).
template <bool MIXED, class Col, class Rec = NoRec>
SHD void icloud(Col& C, const MpConst& K, const MpConstF& KF, bool valid, LevState& S, const LevelStore& P,
                double& qa, const Rec& rec = Rec()) {
  double &qv = S.qv, &ql = S.ql, &qr = S.qr, &qi = S.qi, &qs = S.qs, &qg = S.qg, &tz = S.tz;
  double q_liq, q_sol, cvm;
  icloud_melt_freeze(K, qv, ql, qr, qi, qs, qg, tz, P.den, q_liq, q_sol, cvm);
  rec.value(1, qi);
  double di;
  if (K.z_slope_ice) {
    di = mono_slope(C, qi);
    rec.value(0, di);
    di = qmax(di, qmax(QVMIN, P.h_var() * qi));
  } else {
    di = qmax(QVMIN, P.h_var() * qi);
  }
  if (valid) {
    if constexpr (MIXED)
      icloud_processes_m(K, KF, qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac(), P.vtg(), P.vtr(), P.vts(), P.p1(),
                         di, q_liq, q_sol, cvm);
    else
      icloud_processes(K, qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac(), P.vtg(), P.vtr(), P.vts(), P.p1(), di,
                       q_liq, q_sol, cvm);
    rec.state(0, S);
    if constexpr (MIXED)
      subgrid_z_proc<double, float>(K, P.h_var(), P.rh_adj(), P.rh_rain(), qa, qg, qi, ql, qr, qs, qv, tz, P.den,
                                    P.denfac(), P.p1(), &KF);
    else
      subgrid_z_proc(K, P.h_var(), P.rh_adj(), P.rh_rain(), qa, qg, qi, ql, qr, qs, qv, tz, P.den, P.denfac(), P.p1());
  }
}

// ------------------------------------------------------------------ kernel
// The step of columns c0 .. c0 + G - 1 between staging in and staging out,
// on layout LY: inputs are read from, and outputs written to, the tiles at
// `sm` (field f of block column g at level k at (f * G + g) * RP + k);
// `scr` and `work` are the barrier groups' scratch and work rows. Every
// thread of a barrier group runs the whole step, idle ones (levels beyond L,
// columns beyond the domain, a packed group's idle tail) with valid false,
// so that the groups' vertical operations see all their threads.
// MIXED selects the mixed-precision process rates (mp_physics_mixed.cuh).
template <class LY, bool MIXED, bool FLAGS = false>
SHD void mp_body(const MpArgs& A, double* sm, double* scr, double* work, const int64_t c0) {
  constexpr int RP = LY::RP;
  constexpr int G = LY::G;
  const MpConst& K = A.K;
  const MpConstF& KF = A.KF;
  const int L = A.nz;
  typename LY::Col C;
  const int g = LY::setup(C, threadIdx.x, L, scr, work);
  const bool slot_ok = g < G;
  const int64_t col = c0 + (slot_ok ? g : 0);
  const bool col_ok = slot_ok && col < A.ncol;
  const int k = C.k;
  const bool valid = col_ok && k < L;
  double* tile = sm + (size_t)(slot_ok ? g : 0) * RP + (valid ? k : 0);  // field f of this level at tile[f * G * RP]
  auto TL = [&](int f) -> double& { return tile[(size_t)f * G * RP]; };

  const int64_t cc = col < A.ncol ? col : A.ncol - 1;
  const int64_t cj = div_nx(A, cc), ci = cc - cj * A.nx;
  LevState S;
  LevelStore P;
  P.den = 1.0;
  // ------------------------------------------------ fields_init (:27-276)
  fields_init(C, K, valid, valid ? TL(IN_PT) : 250.0, valid ? TL(IN_QV) : 0.0, valid ? TL(IN_QL) : 0.0,
              valid ? TL(IN_QR) : 0.0, valid ? TL(IN_QI) : 0.0, valid ? TL(IN_QS) : 0.0, valid ? TL(IN_QG) : 0.0,
              valid ? TL(IN_DELP) : 1.0, valid ? TL(IN_W) : 0.0, valid ? TL(IN_DELZ) : -100.0,
              A.land.p[ci * A.land.si + cj * A.land.sj], A.area.p[ci * A.area.si + cj * A.area.sj], S, P);

  if (k == L - 1) {
#pragma unroll
    for (int n = CV_RAIN; n <= CV_GRAUPEL; ++n) C.cv[n] = 0.0;
  }
#pragma unroll 1
  for (int it = 0; it < K.ntimes; ++it) {
    unsigned fl = 0u;  // this sub-step's column flags (FLAGS only)
    // warm_rain with is_first, sedimentation, warm_rain again (one copy
    // of the warm_rain code, run twice)
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      const bool is_first = pass == 0;
      if (is_first) substep_geometry(C, K, valid, valid ? TL(IN_PT) : 250.0, valid ? TL(IN_DELZ) : -100.0, S, P);
      double m1_rain, mp_rain;
      bool falls = false;
      warm_rain<MIXED>(C, K, KF, valid, S, P, m1_rain, mp_rain, FLAGS ? &falls : nullptr);
      if constexpr (FLAGS) fl |= falls ? (is_first ? FLAG_RAIN_FALLS_1 : FLAG_RAIN_FALLS_2) : 0u;
      if (k == L - 1) C.cv[CV_RAIN] += m1_rain;
      P.mp() = is_first ? P.mp() + mp_rain : P.mp() + mp_rain + P.mp_sol();
      if (!is_first) break;
      sedimentation<MIXED>(C, K, KF, valid, S, P, FLAGS ? &fl : nullptr);
    }
    icloud<MIXED>(C, K, KF, valid, S, P, TL(IN_QAZ));  // the accumulator stays in its tile
    if constexpr (FLAGS) {
      if (k == 0 && col_ok) A.flags[(int64_t)it * A.ncol + col] = (int)fl;
    }
  }
  const double qv = S.qv, ql = S.ql, qr = S.qr, qi = S.qi, qs = S.qs, qg = S.qg, tz = S.tz;
  const double dp1 = P.dp1();
  // ------------------------------------------------ fields_update (:1452-1553)
  const double dp0 = valid ? TL(IN_DELP) : 1.0;
  const double u0 = valid ? TL(IN_UA) : 0.0;
  const double v0 = valid ? TL(IN_VA) : 0.0;
  double u1 = u0, v1 = v0;
  if (K.sedi_transport) {
    double au, av, b;
    if (k == 0 || !valid) {
      au = u0;
      av = v0;
      b = 0.0;
    } else {
      const double mp = P.mp();
      const Divisor<double> by_D(dp0 + mp);
      au = by_D(dp0 * u0);
      av = by_D(dp0 * v0);
      b = by_D(mp);
    }
    C.scan_affine2(au, b, av, b, u1, v1);
  }
  if (valid) {
    const double rdt = K.rdt;
    const double omq0 = qdiv(dp0, dp1);
    const double qv0 = TL(IN_QV) * omq0, ql0 = TL(IN_QL) * omq0, qr0 = TL(IN_QR) * omq0;
    const double qi0 = TL(IN_QI) * omq0, qs0 = TL(IN_QS) * omq0, qg0 = TL(IN_QG) * omq0;
    const double t0 = TL(IN_PT), qa0 = TL(IN_QA), qa = TL(IN_QAZ), w = P.w();
    const double omq = qdiv(dp1, dp0);
    const double inc_qv = rdt * (qv - qv0) * omq;
    const double inc_ql = rdt * (ql - ql0) * omq;
    const double inc_qr = rdt * (qr - qr0) * omq;
    const double inc_qi = rdt * (qi - qi0) * omq;
    const double inc_qs = rdt * (qs - qs0) * omq;
    const double inc_qg = rdt * (qg - qg0) * omq;
    const double cvm = K.c_air + qv * K.c_vap + (qr + ql) * K.C_LIQ + (qi + qs + qg) * K.C_ICE;
    const double inc_pt = qdivc(rdt * (tz - t0) * cvm, PH_CP_AIR, 1.0 / PH_CP_AIR);
    const double inc_qa = K.do_qa ? 0.0 : rdt * (qdiv(qa, (double)K.ntimes) - qa0);
    const double inc_u = K.sedi_transport ? (u1 - u0) * rdt : 0.0;
    const double inc_v = K.sedi_transport ? (v1 - v0) * rdt : 0.0;
    TL(OUT_PT_DT) = inc_pt;
    TL(OUT_QV_DT) = inc_qv;
    TL(OUT_QL_DT) = inc_ql;
    TL(OUT_QR_DT) = inc_qr;
    TL(OUT_QI_DT) = inc_qi;
    TL(OUT_QS_DT) = inc_qs;
    TL(OUT_QG_DT) = inc_qg;
    TL(OUT_QA_DT) = inc_qa;
    TL(OUT_UDT) = inc_u;
    TL(OUT_VDT) = inc_v;
    TL(OUT_W) = w;
    TL(OUT_QAZ) = qa;
    // the device error word: the first column (+ 1) that produced a NaN or
    // an infinity, for the host to read after the step (never traps)
    // (x 0 is NaN for an infinity or a NaN, and 0 otherwise)
    double z = inc_pt * 0.0;
    for (const double x : {inc_qv, inc_ql, inc_qr, inc_qi, inc_qs, inc_qg, inc_qa, inc_u, inc_v, w, qa})
      z = __fma_rn(x, 0.0, z);
    if (A.err && !(z == 0.0)) atomicCAS(A.err, 0, (int)(col + 1));
  }
  if (k == L - 1 && col_ok) {
    const double convt = 86400.0 * K.rdt * K.RGRAV;
    const double rain = C.cv[CV_RAIN], ice = C.cv[CV_ICE], snow = C.cv[CV_SNOW], graupel = C.cv[CV_GRAUPEL];
    if (A.rain) A.rain[col] = rain * convt;
    if (A.snow) A.snow[col] = snow * convt;
    if (A.ice) A.ice[col] = ice * convt;
    if (A.graupel) A.graupel[col] = graupel * convt;
    if (A.err && !(isfinite(rain) && isfinite(snow) && isfinite(ice) && isfinite(graupel)))
      atomicCAS(A.err, 0, (int)(col + 1));
  }
}

// One block's work: columns c0 .. c0 + G - 1 of the domain described by A.
template <class LY, bool MIXED, bool FLAGS = false>
SHD void mp_block(const MpArgs& A, double* sm, const int64_t c0) {
  using SM = Smem<LY>;
  stage_in<LY>(A, sm, c0);
  __syncthreads();
  mp_body<LY, MIXED, FLAGS>(A, sm, sm + SM::scratch, sm + SM::work, c0);
  __syncthreads();
  stage_out<LY>(A, sm, c0);
}

template <class LY, int MINB, bool MIXED, bool FLAGS = false>
__global__ void __launch_bounds__(LY::THREADS, MINB) mp_step_kernel(const __grid_constant__ MpArgs A) {
  extern __shared__ double sm[];
  mp_block<LY, MIXED, FLAGS>(A, sm, (int64_t)blockIdx.x * LY::G);
}

// Many domains (ensemble members) in one persistent launch. Work item wi
// of the flattened index space is block (wi - offs[m]) of member m, where
// offs[m] <= wi < offs[m + 1] (offs holds nm + 1 prefix sums of each member's
// ceil(ncol / G)). The persistent blocks take items from a device counter
// (zero at launch), so a block that drew cheap columns takes more of them:
// the items' cost varies with the physics their columns run. A block copies
// its member's parameter block into shared memory when the member changes;
// the step body reads its constants from there. Measured with 64 members
// (C24/C48/C96, L79): a fixed stride of items per block and a prefetch of
// the next item's inputs were both slower.
SHD int find_member(const int64_t* __restrict__ offs, int nm, int64_t wi) {
  int lo = 0, hi = nm - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offs[mid] <= wi)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

template <class LY, int MINB, bool MIXED>
__global__ void __launch_bounds__(LY::THREADS, MINB)
    mp_ensemble_kernel(const MpArgs* __restrict__ members, const int64_t* __restrict__ offs, int nm,
                       unsigned long long* __restrict__ counter) {
  extern __shared__ double sm[];
  __shared__ MpArgs sargs;
  __shared__ long long sitem;
  __shared__ int smember;
  const int64_t total = offs[nm];
  int loaded = -1;
  for (;;) {
    if (threadIdx.x == 0) {
      sitem = (long long)atomicAdd(counter, 1ull);
      smember = sitem < total ? find_member(offs, nm, sitem) : 0;
    }
    __syncthreads();
    const int64_t wi = sitem;
    const int m = smember;
    if (wi >= total) break;
    if (m != loaded) {
      const int* src = reinterpret_cast<const int*>(members + m);
      int* dst = reinterpret_cast<int*>(&sargs);
      constexpr int nwords = (int)(sizeof(MpArgs) / sizeof(int));
      for (int e = threadIdx.x; e < nwords; e += blockDim.x) dst[e] = src[e];
      loaded = m;
      __syncthreads();
    }
    mp_block<LY, MIXED>(sargs, sm, (wi - offs[m]) * LY::G);
    __syncthreads();  // the item is done with sargs, sitem and the tiles
  }
}

// Launch the step over ceil(ncol / G) column blocks.
template <class LY, bool MIXED, bool FLAGS = false>
cudaError_t launch_step(const MpArgs& A, cudaStream_t st) {
  constexpr int G = LY::G;
  auto kern = mp_step_kernel<LY, 1, MIXED, FLAGS>;
  const size_t smem = Smem<LY>::bytes;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)((A.ncol + G - 1) / G), LY::THREADS, smem, st>>>(A);
  return cudaGetLastError();
}

// The first of the layouts (in the order of their columns per block) whose
// blocks fit the SMs in one wave, else the last: the step of a group of warps
// waits on its own FP64 latency, so a domain that leaves SMs idle runs sooner
// with fewer columns per block (144 columns of L79: 33 us with 2 per block,
// 35 with 4, 38 with 6, 41 with 8), while a large one wants the block that
// keeps the SM busiest.
constexpr int B200_SMS = 148;
template <bool MIXED, bool FLAGS, class LY, class... More>
cudaError_t launch_fitting(const MpArgs& A, cudaStream_t st) {
  if constexpr (sizeof...(More) > 0) {
    if (A.ncol > (int64_t)LY::G * B200_SMS) return launch_fitting<MIXED, FLAGS, More...>(A, st);
  }
  return launch_step<LY, MIXED, FLAGS>(A, st);
}

// 65..80 levels (L79): two columns on each group of 5 warps (PackedLayout).
// Every launch of this level range (plain, mixed, flag-recording, ensemble)
// packs two columns per 5 warps, so a column's arithmetic, and with it its
// rounding, is the same in all. Groups per block at C96 L79 (ms per step,
// plain / mixed; the register cap is 65,536 / threads): 3 groups (480
// threads, 128 registers) 2.26 / 1.76, 4 groups (640, 96) 1.89 / 1.38,
// 5 groups (800, 72) 1.98 / 1.43, 6 groups (960, 64) 2.24 / 1.58: beyond 4
// the registers no longer hold the state in use.
constexpr int PACK80_LMIN = 65, PACK80_LMAX = 80;
using Packed80 = PackedLayout<5, 2, 4>;

// The launch for each level range. The widest block of a range holds 24 warps
// (80 registers; six warps per scheduler) where whole columns allow. C96
// (ms, plain / mixed), by columns per block: L31 8: 0.84 / 0.50, 15: 0.82 /
// 0.57, 24: 0.70 / 0.50; L63 8: 1.73 / 1.22, 10: 1.62 / 1.13, 12: 1.57 / 1.09,
// 14: 1.67 / 1.18; L90 4: 2.87 / 2.13, 6: 2.46 / 1.76, 7: 2.36 / 1.68,
// 8: 2.06 / 1.52, 9: 2.19 / 1.55; L127 4: 3.51 / 2.55, 5: 3.30 / 2.36,
// 6: 3.22 / 2.27, 7 (28 warps, 72 registers): 3.16 / 2.19, 8: 3.40 / 2.33.
// At L127 the 7-column block is the faster one only when its waves are many
// (3,233 columns, 4 waves of either: 0.226 against 0.205). These times compare
// the shapes, with the arithmetic of the day; the shapes taken now run L31 in
// 0.71 / 0.50, L63 1.54 / 1.11, L79 1.87 / 1.39, L90 2.01 / 1.55 and L127
// 3.10 / 2.22.
template <bool MIXED, bool FLAGS>
cudaError_t launch_shapes(const MpArgs& A, cudaStream_t st) {
  const int L = A.nz;
  if (L <= 32) return launch_fitting<MIXED, FLAGS, ColumnLayout<1, 8>, ColumnLayout<1, 24>>(A, st);
  if (L <= 64)
    return launch_fitting<MIXED, FLAGS, ColumnLayout<2, 4>, ColumnLayout<2, 8>, ColumnLayout<2, 12>>(A, st);
  if (L <= PACK80_LMAX)
    return launch_fitting<MIXED, FLAGS, PackedLayout<5, 2, 1>, PackedLayout<5, 2, 2>, PackedLayout<5, 2, 3>,
                          Packed80>(A, st);
  if (L <= 96)
    return launch_fitting<MIXED, FLAGS, ColumnLayout<3, 2>, ColumnLayout<3, 4>, ColumnLayout<3, 8>>(A, st);
  if (L <= 128) {
    if (A.ncol > 8 * 7 * B200_SMS) return launch_step<ColumnLayout<4, 7>, MIXED, FLAGS>(A, st);
    return launch_fitting<MIXED, FLAGS, ColumnLayout<4, 2>, ColumnLayout<4, 4>, ColumnLayout<4, 6>>(A, st);
  }
  return launch_fitting<MIXED, FLAGS, ColumnLayout<8, 1>, ColumnLayout<8, 3>>(A, st);
}

// Launch of the ensemble kernel with `grid` persistent blocks; `counter`
// (one word) is zeroed on `st` first.
template <class LY, int MINB, bool MIXED>
cudaError_t launch_ensemble(const MpArgs* members, const int64_t* offs, int nm, unsigned long long* counter, int grid,
                            cudaStream_t st) {
  const size_t smem = Smem<LY>::bytes;
  auto kern = mp_ensemble_kernel<LY, MINB, MIXED>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st)) != cudaSuccess) return e;
  kern<<<grid, LY::THREADS, smem, st>>>(members, offs, nm, counter);
  return cudaGetLastError();
}

}  // namespace SHIELD_ARITH
}  // namespace shield
