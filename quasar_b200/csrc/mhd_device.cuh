// Device numerics of the 2-D ideal-MHD step (sm_100a, FP64).
//
// Pointwise formulas follow the reference's numerics headers formula by
// formula (cited per function, paths relative to the quasar tree) so that the
// result matches its own path to rounding.  The reference evaluates many sums
// through exact-expansion arithmetic (numerics/scaled_arithmetic.hpp).  Here
// ordinary FP64 (with FMA contraction) is used everywhere except at the sites
// where the exact sum creates an exact invariance the algorithm branches on:
// collocating a constant face field returns the constant, and replacing the
// normal field by an equal value leaves the energy bit-identical.  Those sites
// use compensated sums built from non-contracting IEEE intrinsics.
#pragma once

#include <cstdint>

namespace qb {

struct St {
  double rho, mx, my, mz, E, bx, by, bz;
};
struct Pr {
  double rho, vx, vy, vz, p, bx, by, bz;
};
struct Fx {
  double rho, mx, my, mz, E, bx, by, bz;
};

__host__ __device__ inline double comp(const St& s, int c) {
  switch (c) {
    case 0: return s.rho;
    case 1: return s.mx;
    case 2: return s.my;
    case 3: return s.mz;
    case 4: return s.E;
    case 5: return s.bx;
    case 6: return s.by;
    default: return s.bz;
  }
}

constexpr double kEps = 2.220446049250313080847e-16;
constexpr double kTiny = 2.2250738585072014e-308;
constexpr double kInf = __builtin_huge_val();

// ---- compensated sums (never contracted) ---------------------------------
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = __dadd_rn(a, b);
  const double bb = __dadd_rn(s, -a);
  e = __dadd_rn(__dadd_rn(a, -__dadd_rn(s, -bb)), __dadd_rn(b, -bb));
}
// Correctly rounded (up to rare ties) a+b+c of already rounded terms.
__device__ __forceinline__ double crsum3(double a, double b, double c) {
  double s, e1, e2;
  two_sum(a, b, s, e1);
  two_sum(s, c, s, e2);
  return __dadd_rn(s, __dadd_rn(e1, e2));
}
// Sum of exact products w[k]*x[k], rounded once (Dot2).
template <int N>
__device__ __forceinline__ double exact_dot(const double* w, const double* x) {
  double s = __dmul_rn(w[0], x[0]);
  double c = fma(w[0], x[0], -s);
#pragma unroll
  for (int k = 1; k < N; ++k) {
    const double p = __dmul_rn(w[k], x[k]);
    const double pe = fma(w[k], x[k], -p);
    double e;
    two_sum(s, p, s, e);
    c = __dadd_rn(c, __dadd_rn(e, pe));
  }
  return __dadd_rn(s, c);
}

// ---- division by a cell size ----------------------------------------------
// Reciprocal of h when h is a power of two whose reciprocal is a normal
// number (then it is exact), else 0.
__device__ __forceinline__ double pow2_recip(double h) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(h);
  const unsigned e = unsigned(b >> 52) & 0x7ffu;
  const bool pow2 = (b & 0x000fffffffffffffull) == 0ull && e >= 2u && e <= 2044u;
  return pow2 ? 1.0 / h : 0.0;
}
// x / h, formed as x * (1/h) where pow2_recip gave the exact reciprocal rh:
// both are the correctly rounded value of the same real number, so the bits
// are those of the division (every grid whose side is a power-of-two number
// of cells on a unit box takes the multiplication).
__device__ __forceinline__ double div_by(double x, double h, double rh) {
  return rh != 0.0 ? __dmul_rn(x, rh) : __ddiv_rn(x, h);
}

// ---- reciprocal and square root to about one ulp -----------------------------
// The hardware approximation (20 bits) refined once by the cubic member of
// Householder's iterations for 1/x - y and 1/x - y^2 ("The Numerical
// Treatment of a Single Nonlinear Equation", 1970): with e = 1 - x y the
// reciprocal is y (1 + e + e^2) up to e^3 < 2^-59, and with e = 1 - x y^2 the
// inverse square root is y (1 + e/2 + 3 e^2/8).  Three and five FP64
// instructions and no branch, where the correctly rounded forms take twice
// as many and a test for the exceptional operands.  For results that depend
// continuously on rounding, x normal and positive or negative (square root:
// positive); subnormal, infinite and NaN operands give a non-finite value, and
// the reciprocal is zero from 2^1022 on.
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// Densities below the normal range are admissible too, but rcp_nr has NaN for
// them, which every admissibility test refuses; the last resort of each kernel
// (first-order face states, the face-average Riemann problem and its speeds)
// scales them by a power of two.
__device__ __forceinline__ bool subnormal(double x) {
  return unsigned(__double2hiint(x)) < 0x00100000u;
}
__device__ __forceinline__ double rcp_rho(double x) {
  const double z = subnormal(x) ? 0x1p64 : 1.0;
  return rcp_nr(x * z) * z;
}
__device__ __forceinline__ double rsqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// sqrt of finite x >= 0 (x below the normal range: 0).  Infinity gives NaN, as
// infinity times its inverse root: a caller whose operand can overflow tests it.
__device__ __forceinline__ double sqrt_nr(double x) {
  const double s = x * rsqrt_nr(x);
  return x < kTiny ? 0.0 : s;
}

// ---- EOS helpers: numerics/mhd_state.hpp ---------------------------------
// Evaluated without FMA contraction, in the reference's operation order: at a
// degenerate wave fan (zero transverse field) the eigenvector weights are
// square roots of rounding-level differences of these quantities, so their
// bits decide the branch.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double sq3(double x, double y, double z) {
  return add(add(mul(x, x), mul(y, y)), mul(z, z));
}
// Divisions of the functions below, all by a few divisors with several
// numerators each.  PlainDiv: the division operator.
struct PlainDiv {
  struct By {
    double b;
    __device__ __forceinline__ double of(double a) const { return __ddiv_rn(a, b); }
  };
  __device__ __forceinline__ By by(double b) { return By{b}; }
};
// SharedDiv: the same bits from one correctly rounded reciprocal y per divisor
// (two corrections of rcp_nr's operand by its residual; Markstein,
// "Computation of Elementary Functions on the IBM RISC System/6000
// Processor", 1990) and four FP64 instructions a quotient: q0 = RN(a yl + RN(a
// y)), yl the remainder of y, is within an ulp of a / b, its residual a - b q0
// is exact, and RN(q0 + (a - b q0) y) is then the correctly rounded quotient
// (theorem 7.1 there).  The theorem leaves out one significand, all ones,
// whose reciprocal the corrections may leave an ulp off; from the hardware's
// approximation they do not, and the quotients are those of division
// (tests/test_gpu_step_math.py covers that significand).  A divisor outside
// 2^-900 .. 2^900 sets `bad`: the caller repeats the work with PlainDiv.  A
// numerator below 1e-291 may come out an ulp off, in sums that hold a term of
// order one.
struct SharedDiv {
  bool bad = false;
  struct By {
    double b, y, yl;
    __device__ __forceinline__ double of(double a) const {
      const double q = fma(a, yl, __dmul_rn(a, y));
      return fma(fma(-b, q, a), y, q);
    }
  };
  __device__ __forceinline__ By by(double b) {
    bad = bad || ((unsigned(__double2hiint(b)) >> 20) & 0x7ffu) - 123u >= 1800u;
    const double y0 = rcp_nr(b);
    const double y = fma(y0, fma(-b, y0, 1.0), y0);
    return By{b, y, fma(-b, y, 1.0) * y};
  }
};

// mhd_state.hpp:92-100
template <class D>
__device__ __forceinline__ double scaled_norm3(D& dv, double x, double y, double z) {
  const double s = fmax(fabs(x), fmax(fabs(y), fabs(z)));
  if (s == 0.0) return 0.0;
  const auto q = dv.by(s);
  return mul(s, sqrt(sq3(q.of(x), q.of(y), q.of(z))));
}
// mhd_state.hpp:105-114
template <class D>
__device__ __forceinline__ double half_sq3(D& dv, double x, double y, double z) {
  const double s = fmax(fabs(x), fmax(fabs(y), fabs(z)));
  if (s == 0.0) return 0.0;
  const auto q = dv.by(s);
  return mul(mul(0.5, s), mul(s, sq3(q.of(x), q.of(y), q.of(z))));
}
// mhd_state.hpp:118-128, with the quotient by sqrt(rho)
template <class D, class Q>
__device__ __forceinline__ double kin_mom(D& dv, double mx, double my, double mz, const Q& sr) {
  const double s = fmax(fabs(mx), fmax(fabs(my), fabs(mz)));
  if (s == 0.0) return 0.0;
  const auto d = dv.by(s);
  const double q = sr.of(s);
  return mul(mul(0.5, q), mul(q, sq3(d.of(mx), d.of(my), d.of(mz))));
}
__device__ __forceinline__ double scaled_norm3(double x, double y, double z) {
  PlainDiv d;
  return scaled_norm3(d, x, y, z);
}
__device__ __forceinline__ double half_sq3(double x, double y, double z) {
  PlainDiv d;
  return half_sq3(d, x, y, z);
}
__device__ __forceinline__ double kin_mom(double mx, double my, double mz, double rho) {
  PlainDiv d;
  return kin_mom(d, mx, my, mz, d.by(sqrt(rho)));
}
// mhd_state.hpp:131-141
__device__ __forceinline__ double kin_vel(double rho, double vx, double vy, double vz) {
  const double s = fmax(fabs(vx), fmax(fabs(vy), fabs(vz)));
  if (s == 0.0) return 0.0;
  const double q = mul(sqrt(rho), s);
  return mul(mul(0.5, q), mul(q, sq3(vx / s, vy / s, vz / s)));
}
// mhd_state.hpp:148-182, normal Alfven component along x
template <class D, class Q>
__device__ __forceinline__ void magnetosonic(D& dv, const Q& sr, double p, double bn, double bt1,
                                             double bt2, double gamma, double& fast,
                                             double& slow, double& sound, double& can,
                                             double& ca) {
  sound = (p > 0.0 && gamma > 0.0) ? mul(sqrt(gamma), sr.of(sqrt(p))) : 0.0;
  const double ax = sr.of(bn), ay = sr.of(bt1), az = sr.of(bt2);
  ca = scaled_norm3(dv, ax, ay, az);
  can = fabs(ax);
  const double scale = fmax(sound, ca);
  if (!(scale > 0.0)) {
    fast = 0.0;
    slow = 0.0;
    return;
  }
  const auto ds = dv.by(scale);
  const double an = ds.of(sound), bnn = ds.of(ca), cn = ds.of(can);
  const double a2 = mul(an, an), b2 = mul(bnn, bnn), c2 = mul(cn, cn);
  const double sum = add(a2, b2);
  double disc = sub(mul(sum, sum), mul(mul(4.0, a2), c2));
  if (disc < 0.0) disc = 0.0;
  const double f2 = mul(0.5, add(sum, sqrt(disc)));
  const double s2 = (f2 > 0.0) ? mul(a2, c2) / f2 : 0.0;
  fast = mul(scale, sqrt(f2));
  slow = mul(scale, sqrt(s2));
}
// mhd_state.hpp:185-191
template <class D, class Q>
__device__ __forceinline__ double pressure(D& dv, const Q& sr, const St& u, double gamma) {
  const double k = kin_mom(dv, u.mx, u.my, u.mz, sr);
  const double m = half_sq3(dv, u.bx, u.by, u.bz);
  return mul(sub(gamma, 1.0), sub(sub(u.E, k), m));
}
__device__ __forceinline__ double pressure(const St& u, double gamma) {
  PlainDiv d;
  return pressure(d, d.by(sqrt(u.rho)), u, gamma);
}
// Plain-arithmetic EOS for the places whose result depends continuously on
// rounding (Riemann solver, CFL speeds, admissibility tests): one reciprocal
// of rho instead of the reference's component-scaled forms, which only guard
// binary64 overflow for |state| near 1e154 (outside every configuration here).
__device__ __forceinline__ double pressure_f(const St& u, double gamma, double ir) {
  const double k = 0.5 * ((u.mx * u.mx + u.my * u.my + u.mz * u.mz) * ir);
  const double m = 0.5 * (u.bx * u.bx + u.by * u.by + u.bz * u.bz);
  return (gamma - 1.0) * ((u.E - k) - m);
}
// fast magnetosonic speed normal to x from p and 1/rho (mhd_state.hpp:148-182);
// discriminant as (a^2 - b^2)^2 + 4 a^2 b_t^2, free of cancellation
__device__ __forceinline__ double fast_x_f(const St& u, double p, double ir, double gamma) {
  const double a2 = p > 0.0 ? gamma * p * ir : 0.0;
  const double bn2 = u.bx * u.bx * ir;
  const double bt2 = (u.by * u.by + u.bz * u.bz) * ir;
  const double d = a2 - (bn2 + bt2);
  const double disc = d * d + 4.0 * a2 * bt2;
  return sqrt(0.5 * ((a2 + bn2 + bt2) + sqrt(disc)));
}

// Conserved <-> primitive for the limited slopes of the second-order faces,
// whose result depends continuously on rounding: plain arithmetic with one
// reciprocal of rho (igm = 1 / (gamma - 1)) instead of the component-scaled
// forms' seven divisions a state.
__device__ __forceinline__ Pr to_prim(const St& u, double gamma) {
  const double ir = rcp_nr(u.rho);
  return Pr{u.rho, u.mx * ir, u.my * ir, u.mz * ir, pressure_f(u, gamma, ir), u.bx, u.by, u.bz};
}
__device__ __forceinline__ St to_cons(const Pr& w, double igm) {
  const double mx = w.rho * w.vx, my = w.rho * w.vy, mz = w.rho * w.vz;
  return St{w.rho, mx, my, mz,
            w.p * igm + 0.5 * (mx * w.vx + my * w.vy + mz * w.vz) +
                0.5 * (w.bx * w.bx + w.by * w.by + w.bz * w.bz),
            w.bx, w.by, w.bz};
}
// x<->y swap of the in-plane momentum and field (mhd_reconstruct.hip:167-176,
// hlld_core.hpp:45-61).
__device__ __forceinline__ St swap_xy(const St& v) {
  St r = v;
  r.mx = v.my;
  r.my = v.mx;
  r.bx = v.by;
  r.by = v.bx;
  return r;
}

// Admissibility of a face or point state (mhd_reconstruct.hip:414-427,
// mhd_face_quadrature.hpp:68-76), with its pressure supplied.  Every component
// enters the pressure, so with rho finite and positive "p finite and positive"
// already fails for any non-finite component (an infinite momentum or field
// drives p to -inf, an infinite energy to +/-inf, a NaN to NaN): the
// reference's per-component finiteness tests are implied and not repeated,
// the decision is the same.
__device__ __forceinline__ bool point_admissible_p(const St& s, double p) {
  return s.rho > 0.0 && s.rho < kInf && p > 0.0 && p < kInf;
}
__device__ __forceinline__ bool point_admissible_ir(const St& s, double gamma, double ir) {
  return point_admissible_p(s, pressure_f(s, gamma, ir));
}
__device__ __forceinline__ bool point_admissible(const St& s, double gamma) {
  return point_admissible_ir(s, gamma, rcp_nr(s.rho));
}

// The same for a density below the normal range: 2 rho (E - B^2 / 2) > m^2 with
// density, energy and momentum scaled by 2^1000.
__device__ __forceinline__ bool subnormal_admissible(const St& s) {
  constexpr double z = 0x1p1000;
  const double q = 2.0 * (s.E - 0.5 * (s.bx * s.bx + s.by * s.by + s.bz * s.bz));
  const double mx = s.mx * z, my = s.my * z, mz = s.mz * z;
  return subnormal(s.rho) && q < kInf && (s.rho * z) * (q * z) > mx * mx + my * my + mz * mz;
}

__device__ __forceinline__ bool recon_admissible(const St& s, double gamma) {
  return point_admissible(s, gamma);
}

// ---- MP limiter: numerics/mp_limiter.hpp ---------------------------------
__device__ __forceinline__ double minmod2(double a, double b) {
  if (a == 0.0 || b == 0.0 || ((a < 0.0) != (b < 0.0))) return 0.0;
  return (fabs(a) < fabs(b)) ? a : b;
}
__device__ __forceinline__ int sgn(double a) { return a > 0.0 ? 1 : (a < 0.0 ? -1 : 0); }
__device__ __forceinline__ double minmod4(double a, double b, double c, double d) {
  const int sa = sgn(a);
  if (!(sa == sgn(b) && sa == sgn(c) && sa == sgn(d)) || sa == 0) return 0.0;
  const double m = fmin(fmin(fabs(a), fabs(b)), fmin(fabs(c), fabs(d)));
  return sa > 0 ? m : -m;
}
// mp_limiter.hpp:71-148.  `fired` is set when the candidate was changed.
// The normalisations by the local variation and the curvature scale use one
// reciprocal each instead of a division per term (rounding-level difference).
// One window at a time: the form the label pass uses, which needs `fired`.
__device__ __noinline__ double mp_limit(double vl, double vm2, double vm1, double v0,
                                           double vp1, double vp2, bool& fired) {
  const double dmn = v0 - vm1;
  const double dpl = vp1 - v0;
  const double vmp = v0 + minmod2(dpl, 4.0 * dmn);
  const double cc = vl - v0, cm = vl - vmp;
  const bool between = (cc <= 0.0 && cm >= 0.0) || (cc >= 0.0 && cm <= 0.0);
  const double var = fmax(fmax(fabs(dmn), fabs(dpl)), fmax(fabs(cc), fabs(cm)));
  bool roundoff = false;
  if (!between && var > 0.0) {
    const double iv = 1.0 / var;
    roundoff = (fabs(cc) * iv) * (fabs(cm) * iv) <= 1e-10;
  }
  if (between || roundoff) {
    fired = false;
    return vl;
  }
  fired = true;
  const double dm = (vm2 - vm1) - (vm1 - v0);
  const double d0 = (vm1 - v0) - (v0 - vp1);
  const double dp = (v0 - vp1) - (vp1 - vp2);
  const double cs = fmax(fabs(dm), fmax(fabs(d0), fabs(dp)));
  double d4ph = 0.0, d4mh = 0.0;
  if (cs > 0.0) {
    const double ic = 1.0 / cs;
    const double dms = dm * ic, d0s = d0 * ic, dps = dp * ic;
    d4ph = cs * minmod4(4.0 * d0s - dps, 4.0 * dps - d0s, d0s, dps);
    d4mh = cs * minmod4(4.0 * d0s - dms, 4.0 * dms - d0s, d0s, dms);
  }
  const double v_ul = v0 + 4.0 * dmn;
  const double v_av = 0.5 * v0 + 0.5 * vp1;
  const double v_md = v_av - 0.5 * d4ph;
  const double v_lc = v0 + 0.5 * dmn + (4.0 / 3.0) * d4mh;
  const double vmin = fmax(fmin(fmin(v0, vp1), v_md), fmin(fmin(v0, v_ul), v_lc));
  const double vmax = fmin(fmax(fmax(v0, vp1), v_md), fmax(fmax(v0, v_ul), v_lc));
  return vl + minmod2(vmin - vl, vmax - vl);
}
// mp_limiter.hpp:182-224: the unlimited MP interpolation of the W-point
// stencil v[0..W-1] to the face, W = 5 (MP5) or 7 (MP7).  The reference
// divides every term by the stencil's largest magnitude first, which only
// guards binary64 overflow for values near 1e305 (outside every
// configuration here); the weights are applied directly, summed as a shallow
// tree (two-term FMA pairs) rather than one dependent chain, a
// rounding-level difference.
template <int W>
__device__ __forceinline__ double mp_interp_plain(const double* v) {
  if (W == 5) {
    const double a = fma(-13.0, v[1], 2.0 * v[0]);
    const double b = fma(27.0, v[3], 47.0 * v[2]);
    return ((a + b) + (-3.0 * v[4])) * (1.0 / 60.0);
  }
  const double a = fma(25.0, v[1], -3.0 * v[0]);
  const double b = fma(319.0, v[3], -101.0 * v[2]);
  const double c = fma(-38.0, v[5], 214.0 * v[4]);
  return ((a + b) + (c + 4.0 * v[6])) * (1.0 / 420.0);
}

template <int W>
__device__ __forceinline__ double mp_recon(const double* v, bool& fired) {
  const double vl = mp_interp_plain<W>(v);
  constexpr int o = W == 5 ? 0 : 1;
  return mp_limit(vl, v[o], v[o + 1], v[o + 2], v[o + 3], v[o + 4], fired);
}

// ---- both face states of one characteristic variable ----------------------
// x with its sign flipped where the bit `s` (0 or 0x80000000) is set.
__device__ __forceinline__ double flip_sign(double x, int s) {
  return __hiloint2double(__double2hiint(x) ^ s, __double2loint(x));
}
// minmod4(4 p - q, 4 q - p, p, q): with m and M the smaller and larger of |p|
// and |q|, and p, q of one sign, the smallest argument is min(m, 4 m - M)
// (4 M - m >= 3 M), zero if that is negative.
__device__ __forceinline__ double mp_curvature(double p, double q) {
  const double P = fabs(p), Q = fabs(q);
  const bool lt = P < Q;
  const double m = lt ? P : Q, M = lt ? Q : P;
  const double t = fma(4.0, m, -M);
  const double r = t < m ? t : m;
  const bool ok = (__double2hiint(p) ^ __double2hiint(q)) >= 0 && __double2hiint(r) >= 0;
  return ok ? flip_sign(r, __double2hiint(p) & 0x80000000) : 0.0;
}
// One side of mp_limiter.hpp:71-148 in coordinates relative to its centre
// sample and flipped so that the unlimited offset cc is positive: dpl = vp1 -
// v0, dmn = v0 - vm1, md and lc the median and large-curvature offsets.  In
// these coordinates the lower limit is <= 0 <= the upper limit, so only the
// upper one, min(max(dpl, md), max(4 dmn, lc)) or zero, can bind; it is at
// least minmod(dpl, 4 dmn), so the early accept never changes the value and
// only its round-off form is tested, |cc| |cm| <= 1e-10 var^2.  Of var's
// four terms the two differences suffice: |cc| or |cm| is the largest only
// where cc or cm is within 1e-10 of zero relative to a difference, and there
// the limited and the unlimited value agree to that.  An offset whose square
// would leave the binary64 range (below 2^-480, from 2^490) is first scaled, with
// the differences, by a power of two, so that the test is the same at every
// magnitude.  Returns the limited offset.  NaN offsets compare false and are
// returned.
__device__ __forceinline__ double mp_side(double cc, double dpl, double dmn, double md,
                                          double lc) {
  const int s = __double2hiint(cc) & 0x80000000;
  const double ac = fabs(cc);
  const double d = flip_sign(dpl, s), ul = flip_sign(4.0 * dmn, s);
  const double m = flip_sign(md, s), c = flip_sign(lc, s);
  const double A = d > m ? d : m, B = ul > c ? ul : c;
  double bound = A < B ? A : B;
  bound = __double2hiint(bound) < 0 ? 0.0 : bound;
  double mm = fabs(d) < fabs(ul) ? d : ul;
  mm = (__double2hiint(d) ^ __double2hiint(ul)) < 0 ? 0.0 : mm;
  if (!(ac > bound)) return cc;
  double x = ac, y = ac - mm, p = dpl, q = dmn;
  if (unsigned(__double2hiint(ac)) - (543u << 20) >= 970u << 20) {
    const double z = __hiloint2double(__double2hiint(ac) < (543 << 20) ? 1623 << 20 : 423 << 20, 0);
    x *= z;
    y *= z;
    p *= z;
    q *= z;
  }
  const double P = x * y * 1e10;
  const int above = __double2hiint(fma(q, q, -P)) & __double2hiint(fma(p, p, -P));
  return above < 0 ? flip_sign(bound, s) : cc;
}
// The MP5 / MP7 face values on both sides of the face between samples H and
// H + 1 of c[0 .. 2H + 1] (mp_limiter.hpp:71-224 for the window and its
// mirror image).  Everything is formed from the first differences, which
// the two sides share, as are the second differences and the median's
// curvature; the interpolation weights are those of mp_interp_plain summed
// onto the differences.  63 FP64 instructions at MP7 for the pair, where two
// separate windows took about 180 with four divisions.
template <int W>
__device__ __forceinline__ void mp_pair_limit(const double* c, double& wl, double& wr) {
  constexpr int H = W / 2;
  double d[W];
#pragma unroll
  for (int k = 0; k < W; ++k) d[k] = c[k + 1] - c[k];
  double cl, cr;
  if (W == 5) {
    constexpr double q = 1.0 / 60.0;
    cl = fma(24.0 * q, d[2], fma(-2.0 * q, d[0], fma(11.0 * q, d[1], (-3.0 * q) * d[3])));
    cr = -fma(24.0 * q, d[2], fma(-2.0 * q, d[4], fma(11.0 * q, d[3], (-3.0 * q) * d[1])));
  } else {
    constexpr double q = 1.0 / 420.0;
    cl = fma(180.0 * q, d[3], fma(79.0 * q, d[2], (-34.0 * q) * d[4])) +
         fma(-22.0 * q, d[1], fma(3.0 * q, d[0], (4.0 * q) * d[5]));
    cr = -(fma(180.0 * q, d[3], fma(79.0 * q, d[4], (-34.0 * q) * d[2])) +
           fma(-22.0 * q, d[5], fma(3.0 * q, d[6], (4.0 * q) * d[1])));
  }
  const double dm = d[H - 1], d0 = d[H], dp = d[H + 1];
  const double s1 = dm - d[H - 2], s2 = d0 - dm, s3 = dp - d0, s4 = d[H + 2] - dp;
  const double ph = mp_curvature(s2, s3), hd = 0.5 * d0;
  const double ml = mp_curvature(s2, s1), mr = mp_curvature(s3, s4);
  wl = c[H] + mp_side(cl, d0, dm, fma(-0.5, ph, hd), fma(4.0 / 3.0, ml, 0.5 * dm));
  wr = c[H + 1] + mp_side(cr, -d0, -dp, fma(-0.5, ph, -hd), fma(4.0 / 3.0, mr, -0.5 * dp));
}

// ---- HLLD: numerics/hlld_core.hpp ----------------------------------------
// hlld_core.hpp:123-153, from the state, its pressure and 1/rho
__device__ __forceinline__ Fx physical_flux_xp(const St& u, double p, double ir) {
  const double vx = u.mx * ir, vy = u.my * ir, vz = u.mz * ir;
  const double hbn = 0.5 * (u.bx * u.bx);
  const double hbt = 0.5 * (u.by * u.by + u.bz * u.bz);
  Fx f;
  f.rho = u.mx;
  f.mx = u.mx * vx + p + u.by * (0.5 * u.by) + u.bz * (0.5 * u.bz) + u.bx * (-0.5 * u.bx);
  f.my = u.mx * vy + u.bx * (-u.by);
  f.mz = u.mx * vz + u.bx * (-u.bz);
  const double h = ((u.E - hbn) + p) + hbt;
  const double tvb = vy * u.by + vz * u.bz;
  f.E = vx * h + u.bx * (-tvb);
  f.bx = 0.0;
  f.by = u.by * vx + u.bx * (-vy);
  f.bz = u.bz * vx + u.bx * (-vz);
  return f;
}
__device__ __forceinline__ Fx physical_flux_x(const St& u, double gamma) {
  const double ir = 1.0 / u.rho;
  return physical_flux_xp(u, pressure_f(u, gamma, ir), ir);
}
// hlld_core.hpp:157-192
__device__ __noinline__ Fx hll_flux_x(const St& L, const St& R, double sl, double sr,
                                      double gamma) {
  const Fx fl = physical_flux_x(L, gamma);
  const Fx fr = physical_flux_x(R, gamma);
  if (sl >= 0.0) return fl;
  if (sr <= 0.0) return fr;
  const double ss = fmax(fabs(sl), fabs(sr));
  if (!(ss > 0.0) || !isfinite(ss)) return fl;
  const double sln = sl / ss, srn = sr / ss;
  const double den = srn - sln;
  if (!(den > 0.0) || !isfinite(den)) return fl;
  const double wl = srn / den, wr = -sln / den;
  const double dis = ss * (sln * srn / den);
  Fx f;
  f.rho = wl * fl.rho + wr * fr.rho + dis * (R.rho - L.rho);
  f.mx = wl * fl.mx + wr * fr.mx + dis * (R.mx - L.mx);
  f.my = wl * fl.my + wr * fr.my + dis * (R.my - L.my);
  f.mz = wl * fl.mz + wr * fr.mz + dis * (R.mz - L.mz);
  f.E = wl * fl.E + wr * fr.E + dis * (R.E - L.E);
  f.bx = 0.0;
  f.by = wl * fl.by + wr * fr.by + dis * (R.by - L.by);
  f.bz = wl * fl.bz + wr * fr.bz + dis * (R.bz - L.bz);
  return f;
}
// hlld_core.hpp:200-210
__device__ __forceinline__ Fx lf_flux_x(const St& L, const St& R, double gamma) {
  const double irl = 1.0 / L.rho, irr = 1.0 / R.rho;
  const double aL = fabs(L.mx * irl) + fast_x_f(L, pressure_f(L, gamma, irl), irl, gamma);
  const double aR = fabs(R.mx * irr) + fast_x_f(R, pressure_f(R, gamma, irr), irr, gamma);
  const double a = (aL > aR) ? aL : aR;
  return hll_flux_x(L, R, -a, a, gamma);
}
__device__ __forceinline__ bool same_state(const St& a, const St& b) {
  return a.rho == b.rho && a.mx == b.mx && a.my == b.my && a.mz == b.mz && a.E == b.E &&
         a.bx == b.bx && a.by == b.by && a.bz == b.bz;
}

// hlld_core.hpp:213-457 (B0 inactive), with the reciprocal densities and the
// pressures of the two states supplied (the normal-field average leaves the
// gas pressure as it is).  Written for the instruction count, which is what
// bounds the face flux: reciprocals and square roots by rcp_nr / rsqrt_nr,
// the energy and the Alfven speed formed on the upwind side only, one exit to
// the HLL flux for every unresolved case, and the star-region flux in its
// closed form.  By the jump conditions that define them, F + s (U* - U) and
// F* + s* (U** - U*) (the reference's sums) equal the physical flux of the
// star state under the star total pressure p*: rho* s_M, rho* s_M^2 + p* -
// B_n^2, rho* s_M v_t - B_n B_t, s_M B_t - B_n v_t and s_M (E + p*) - B_n
// (v . B); the two differ by rounding.  Star values are formed as the outer
// value plus a correction that vanishes with the jump, so a linear wave's
// flux carries less rounding noise than quotients of whole sums.  Measured
// with the shortcut-free point recovery (wsum) on a flow without uniform
// regions at 2048^2 MP7: face flux 9.6 -> 6.1 ms per step.
// SAME: return the physical flux of two states that agree in every component
// bit for bit (a caller that knows where they do passes false).
template <bool SAME = true>
__device__ __forceinline__ Fx hlld_flux_x(const St& L, const St& R, double gamma, double irl,
                                          double irr, double pL, double pR) {
  if (SAME && same_state(L, R)) return physical_flux_xp(L, pL, irl);
  const double rel = 64.0 * kEps;
  const double bn = 0.5 * L.bx + 0.5 * R.bx, bn2 = bn * bn, hbn2 = 0.5 * bn2;
  const double EL = (L.E - 0.5 * (L.bx * L.bx)) + hbn2;
  const double ER = (R.E - 0.5 * (R.bx * R.bx)) + hbn2;
  const double vxL = L.mx * irl, vxR = R.mx * irr;
  const double btL2 = L.by * L.by + L.bz * L.bz, btR2 = R.by * R.by + R.bz * R.bz;
  const double ptL = pL + (hbn2 + 0.5 * btL2), ptR = pR + (hbn2 + 0.5 * btR2);
  // fast speed squared of each side (fast_x_f); one square root of the larger
  auto fast2 = [&](double p, double ir, double bt2) {
    const double a2 = p > 0.0 ? gamma * p * ir : 0.0;
    const double b2 = bt2 * ir, n2 = bn2 * ir, d = a2 - (n2 + b2);
    return 0.5 * ((a2 + n2 + b2) + sqrt_nr(d * d + 4.0 * a2 * b2));
  };
  const double fL = fast2(pL, irl, btL2), fR = fast2(pR, irr, btR2);
  // an overflowing discriminant leaves NaN on its side, which a maximum would
  // drop: infinite wave speeds, which only the HLL exit takes
  const double cf = fL < kInf && fR < kInf ? sqrt_nr(fL > fR ? fL : fR) : kInf;
  const double sl = (vxL < vxR ? vxL : vxR) - cf, sr = (vxL > vxR ? vxL : vxR) + cf;
  if (sl >= 0.0 || sr <= 0.0) {
    const bool l = sl >= 0.0;
    const St u{l ? L.rho : R.rho, l ? L.mx : R.mx, l ? L.my : R.my, l ? L.mz : R.mz,
               l ? EL : ER,       bn,              l ? L.by : R.by, l ? L.bz : R.bz};
    return physical_flux_xp(u, l ? pL : pR, l ? irl : irr);
  }
  // a_R >= 0 >= a_L by construction, so the difference is never cancelled
  const double dvL = sl - vxL, dvR = sr - vxR;
  const double aL = dvL * L.rho, aR = dvR * R.rho;
  const double idM = rcp_nr(aR - aL);
  const double sm = ((aR * vxR - aL * vxL) + (ptL - ptR)) * idM;
  const double dLs = sl - sm, dRs = sr - sm;
  const double ws = rel * (fabs(sl) + fabs(sr) + fabs(sm) + kTiny);
  const double iL = rcp_nr(dLs), iR = rcp_nr(dRs);
  // single-star states (hlld_core.hpp:306-346), each as the outer value plus a
  // term proportional to s_M - v_n
  const double dmL = sm - vxL, dmR = sm - vxR;
  const double rhoL = fma(L.rho * dmL, iL, L.rho), rhoR = fma(R.rho * dmR, iR, R.rho);
  const double tL = aL * dLs, tR = aR * dRs;
  const double denL = tL - bn2, denR = tR - bn2;
  // (comparisons written so that a NaN is not resolved)
  const bool resolved = fabs(dLs) > ws && fabs(dRs) > ws && rhoL > 0.0 && rhoR > 0.0 &&
                        fabs(denL) > rel * (fabs(tL) + bn2 + kTiny) &&
                        fabs(denR) > rel * (fabs(tR) + bn2 + kTiny);
  const double kL = dmL * rcp_nr(denL), kR = dmR * rcp_nr(denR);
  const double fcL = bn * kL, fcR = bn * kR, bcL = aL * kL, bcR = aR * kR;
  const double vyL0 = L.my * irl, vzL0 = L.mz * irl, vyR0 = R.my * irr, vzR0 = R.mz * irr;
  const double vyL = vyL0 - L.by * fcL, vzL = vzL0 - L.bz * fcL;
  const double vyR = vyR0 - R.by * fcR, vzR = vzR0 - R.bz * fcR;
  const double byL = fma(L.by, bcL, L.by), bzL = fma(L.bz, bcL, L.bz);
  const double byR = fma(R.by, bcR, R.by), bzR = fma(R.bz, bcR, R.bz);
  const double rqL = rsqrt_nr(rhoL), rqR = rsqrt_nr(rhoR);
  // the upwind side of the contact
  const bool l = sm >= 0.0;
  const double a = l ? aL : aR, dm = l ? dmL : dmR, pt = l ? ptL : ptR, vx = l ? vxL : vxR;
  const double pts = fma(a, dm, pt);
  const bool negl = bn2 <= rel * (fabs(pts) + fabs(ptL) + fabs(ptR) + kTiny);
  const double rho = l ? rhoL : rhoR;
  double vy = l ? vyL : vyR, vz = l ? vzL : vzR, by = l ? byL : byR, bz = l ? bzL : bzR;
  const double vb = bn * vx + ((l ? vyL0 : vyR0) * (l ? L.by : R.by) +
                               (l ? vzL0 : vzR0) * (l ? L.bz : R.bz));
  double vbs = sm * bn + (vy * by + vz * bz);
  double E = l ? EL : ER;
  E = fma(dm * (E + fma(a, sm, pt)) + bn * (vb - vbs), l ? iL : iR, E);
  // double-star states (hlld_core.hpp:379-411) inside the Alfven waves
  const double ca = fabs(bn) * (l ? rqL : rqR);
  if (!negl && (l ? sm < ca : sm >= -ca)) {
    const double sqL = rhoL * rqL, sqR = rhoR * rqR;
    const double isum = rcp_nr(sqL + sqR), qq = sqL * sqR;
    const double sg = bn >= 0.0 ? 1.0 : -1.0;
    const double dvy = vyR - vyL, dvz = vzR - vzL, dby = byR - byL, dbz = bzR - bzL;
    const double vyss = fma(sqR * dvy + dby * sg, isum, vyL);
    const double vzss = fma(sqR * dvz + dbz * sg, isum, vzL);
    const double byss = fma(sqL * dby + qq * dvy * sg, isum, byL);
    const double bzss = fma(sqL * dbz + qq * dvz * sg, isum, bzL);
    const double vbss = sm * bn + (vyss * byss + vzss * bzss);
    const double q = l ? -sqL : sqR;
    E = E + q * sg * (vbs - vbss);
    vy = vyss;
    vz = vzss;
    by = byss;
    bz = bzss;
    vbs = vbss;
  }
  const double m = rho * sm;
  Fx f;
  f.rho = m;
  f.mx = m * sm + (pts - bn2);
  f.my = m * vy - bn * by;
  f.mz = m * vz - bn * bz;
  f.E = sm * (E + pts) - bn * vbs;
  f.bx = 0.0;
  f.by = sm * by - bn * vy;
  f.bz = sm * bz - bn * vz;
  // every star quantity enters the energy flux, so a non-finite one shows there
  if (!resolved || !(fabs(f.E + f.rho) < kInf)) {
    const St l2{L.rho, L.mx, L.my, L.mz, EL, bn, L.by, L.bz};
    const St r2{R.rho, R.mx, R.my, R.mz, ER, bn, R.by, R.bz};
    return hll_flux_x(l2, r2, sl, sr, gamma);
  }
  return f;
}
// Face-normal Riemann flux in the lab frame (mhd_face_quadrature.hpp:173-185),
// irl / irr = 1 / rho and pl / pr = pressure of the two states.
template <int DIR, bool SAME = true>
__device__ __forceinline__ Fx riemann(const St& l, const St& r, bool lf, double gamma,
                                      double irl, double irr, double pl, double pr) {
  const St a = DIR == 0 ? l : swap_xy(l);
  const St b = DIR == 0 ? r : swap_xy(r);
  Fx f = lf ? lf_flux_x(a, b, gamma) : hlld_flux_x<SAME>(a, b, gamma, irl, irr, pl, pr);
  if (DIR == 1) {
    const double t = f.mx;
    f.mx = f.my;
    f.my = t;
    const double u = f.bx;
    f.bx = f.by;
    f.by = u;
  }
  return f;
}
template <int DIR>
__device__ __forceinline__ Fx riemann(const St& l, const St& r, bool lf, double gamma) {
  const double irl = 1.0 / l.rho, irr = 1.0 / r.rho;
  return riemann<DIR>(l, r, lf, gamma, irl, irr, pressure_f(l, gamma, irl),
                      pressure_f(r, gamma, irr));
}

// ---- transverse quadrature: numerics/finite_volume_quadrature.hpp:12-68 --
__constant__ double c_gauss3[3] = {5.0 / 18.0, 4.0 / 9.0, 5.0 / 18.0};
__constant__ double c_gauss4[4] = {0.173927422568726925, 0.326072577431273103,
                                   0.326072577431273103, 0.173927422568726925};
__constant__ double c_point5[3][5] = {
    {-0.0392523473402346598, 0.312987195324173573, 0.910833333333333384,
     -0.216320528657506839, 0.0317523473402346601},
    {0.00468749999999999983, -0.0604166666666666671, 1.11145833333333344,
     -0.0604166666666666671, 0.00468749999999999983},
    {0.0317523473402346601, -0.216320528657506839, 0.910833333333333384,
     0.312987195324173573, -0.0392523473402346598}};
__constant__ double c_point7[4][7] = {
    {0.00860109764472105458, -0.0796691475531970394, 0.415576982717296983,
     0.849155569794037945, -0.245805403605616202, 0.0591434746546156687,
     -0.0070025736518584264},
    {0.00327670662777140203, -0.0266359260617751309, 0.0928282644451935562,
     1.08046056237311472, -0.183384586025290314, 0.0375843394851378479,
     -0.00412936084415200903},
    {-0.00412936084415200903, 0.0375843394851378479, -0.183384586025290314,
     1.08046056237311472, 0.0928282644451935562, -0.0266359260617751309,
     0.00327670662777140203},
    {-0.0070025736518584264, 0.0591434746546156687, -0.245805403605616202,
     0.849155569794037945, 0.415576982717296983, -0.0796691475531970394,
     0.00860109764472105458}};

// Weighted sum whose weights add up to one, as the centre sample plus the
// weighted differences from it: samples that all equal the centre one return
// it unchanged, as the reference's explicit shortcut does
// (finite_volume_quadrature.hpp:55-68), without the N - 1 comparisons (which
// issue on the FP64 pipe) or a branch.  Operations and their order are fixed,
// so every kernel forms the same bits.
template <int N>
__device__ __forceinline__ double wsum_diff(const double* w, const double* d, double ref) {
  double acc = 0.0;
#pragma unroll
  for (int t = 0; t < N; ++t)
    if (t != N / 2) acc = t == 0 ? __dmul_rn(w[0], d[0]) : fma(w[t], d[t], acc);
  return __dadd_rn(ref, acc);
}
template <int N>
__device__ __forceinline__ void centre_diff(const double* s, double* d) {
#pragma unroll
  for (int t = 0; t < N; ++t) d[t] = t == N / 2 ? 0.0 : __dsub_rn(s[t], s[N / 2]);
}
template <int N>
__device__ __forceinline__ double wsum(const double* w, const double* s) {
  double d[N];
  centre_diff<N>(s, d);
  return wsum_diff<N>(w, d, s[N / 2]);
}

// Compile-time selected quadrature weights (constant-bank operands).
template <int ORDER>
__device__ __forceinline__ double point_w(int q, int t) {
  return ORDER == 5 ? c_point5[q][t] : c_point7[q][t];
}
template <int ORDER>
__device__ __forceinline__ double gauss_w(int q) {
  return ORDER == 5 ? c_gauss3[q] : c_gauss4[q];
}
// Point value at Gauss node q from N = 5/7 transverse averages s[].
template <int ORDER>
__device__ __forceinline__ double point_value(int q, const double* s) {
  constexpr int N = ORDER == 5 ? 5 : 7;
  double w[N];
#pragma unroll
  for (int t = 0; t < N; ++t) w[t] = point_w<ORDER>(q, t);
  return wsum<N>(w, s);
}
// Point values at all Q = 3/4 Gauss nodes from the same N transverse
// averages.  The nodes lie symmetrically about the centre, node Q - 1 - q with
// node q's weights reversed, so a pair of nodes is centre + A +- B with A from
// the even and B from the odd differences of the samples at distance k:
// 27 FP64 instructions for four nodes of seven samples where four separate
// sums take 34.  Equal samples return their value (every difference is zero).
// wE / wO: half the sum and half the difference of node q's weights at k, -k.
template <int ORDER>
__device__ __forceinline__ void point_values(const double* s, double* out) {
  constexpr int H = ORDER == 5 ? 2 : 3, Q = ORDER == 5 ? 3 : 4;
  constexpr double wE5[2][2] = {{0.5 * (-0.216320528657506839 + 0.312987195324173573),
                                 0.5 * (0.0317523473402346601 - 0.0392523473402346598)},
                                {-0.0604166666666666671, 0.00468749999999999983}};
  constexpr double wO5[2][2] = {{0.5 * (-0.216320528657506839 - 0.312987195324173573),
                                 0.5 * (0.0317523473402346601 + 0.0392523473402346598)},
                                {0.0, 0.0}};
  constexpr double wE7[2][3] = {{0.5 * (-0.245805403605616202 + 0.415576982717296983),
                                 0.5 * (0.0591434746546156687 - 0.0796691475531970394),
                                 0.5 * (-0.0070025736518584264 + 0.00860109764472105458)},
                                {0.5 * (-0.183384586025290314 + 0.0928282644451935562),
                                 0.5 * (0.0375843394851378479 - 0.0266359260617751309),
                                 0.5 * (-0.00412936084415200903 + 0.00327670662777140203)}};
  constexpr double wO7[2][3] = {{0.5 * (-0.245805403605616202 - 0.415576982717296983),
                                 0.5 * (0.0591434746546156687 + 0.0796691475531970394),
                                 0.5 * (-0.0070025736518584264 - 0.00860109764472105458)},
                                {0.5 * (-0.183384586025290314 - 0.0928282644451935562),
                                 0.5 * (0.0375843394851378479 + 0.0266359260617751309),
                                 0.5 * (-0.00412936084415200903 - 0.00327670662777140203)}};
  const double ref = s[H];
  double e[H], o[H];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    e[k] = fma(-2.0, ref, __dadd_rn(s[H + 1 + k], s[H - 1 - k]));
    o[k] = __dsub_rn(s[H + 1 + k], s[H - 1 - k]);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double* we = ORDER == 5 ? wE5[q] : wE7[q];
    const double* wo = ORDER == 5 ? wO5[q] : wO7[q];
    double A = __dmul_rn(we[0], e[0]), B = __dmul_rn(wo[0], o[0]);
#pragma unroll
    for (int k = 1; k < H; ++k) {
      A = fma(we[k], e[k], A);
      B = fma(wo[k], o[k], B);
    }
    const double m = __dadd_rn(ref, A);
    if (ORDER == 5 && q == 1) {
      out[1] = m;  // the centre node
    } else {
      out[q] = __dadd_rn(m, B);
      out[Q - 1 - q] = __dsub_rn(m, B);
    }
  }
}
// Gauss average of Q = 3/4 point values.
template <int ORDER>
__device__ __forceinline__ double gauss_avg(const double* s) {
  constexpr int Q = ORDER == 5 ? 3 : 4;
  double w[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) w[q] = gauss_w<ORDER>(q);
  return wsum<Q>(w, s);
}

}  // namespace qb
