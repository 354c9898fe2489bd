// sm_100a kernels of the 2-D ideal-MHD SSP-RK3 step (FP64).
//
// One RK stage is a short pipeline of grid-wide kernels whose intermediates
// round-trip through L2/HBM (the step is FP64-compute-bound, so the extra
// traffic is cheap next to the recomputation a fully fused tile would need):
//
//   colloc_check   cell-collocated B of the stage input (computed once per
//                  state instead of once per load) + admissibility of the
//                  previous candidate + preflights of the live state
//   reconstruct    MP5/MP7 characteristic L/R face states, one face/thread
//   face_flux      Gauss-point HLLD -> face flux, face E_z (the same solve),
//                  no-jump proof and, on stage 0, the CFL signal speed
//   cell_emf       cell-average E_z + (stage 0) the dt max-reduction
//   corner_emf     upwind CT corner E_z
//   update         flux difference + EMF curl + Shu-Osher combine, fused
//   fill_ghosts    boundary closure of the new state
//
// dt lives in device memory: the stage-0 update reads it, so a whole step
// (or many) runs without a host round trip and can be captured in a graph.
#include "mhd_device.cuh"
#include "mhd_kernels.cuh"
#include "tc.cuh"

#include <cudaTypedefs.h>

#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>

#include <algorithm>
#include <mutex>
#include <vector>

namespace qb {

namespace cg = cooperative_groups;

namespace {

constexpr int kBX = 32;  // block x (coalesced along i)


// Corner/face-table index map (reference mhd_ct.hip:126-139): periodic axes
// wrap into [0,n); physical sides clamp into [0,n].
__device__ __forceinline__ int face_index(int q, int n, int lo, int hi) {
  if (lo == 0 && hi == 0) {
    int w = q % n;
    if (w < 0) w += n;
    return w;
  }
  if (q < 0) return 0;
  if (q > n) return n;
  return q;
}

__device__ __forceinline__ bool in_pad(const Grid& g, int i, int j) {
  return i >= -g.ng && i < g.nx + g.ng && j >= -g.ng && j < g.ny + g.ng;
}

// Cell state with the high-order collocated field (reference
// mhd_staggering.hpp:321-338, collocation order 0).
__device__ __forceinline__ St load_cell(const StateP& u, long long k) {
  return St{__ldg(u.c[0] + k), __ldg(u.c[1] + k), __ldg(u.c[2] + k), __ldg(u.c[3] + k),
            __ldg(u.c[4] + k), __ldg(u.bxc + k), __ldg(u.byc + k), __ldg(u.c[7] + k)};
}

// Two-face average used by the low-order retry operator
// (mhd_staggering.hpp:243-254): the outermost high ghost keeps its sole face.
__device__ __forceinline__ double low_order_b(const double* f, const Grid& g, int cell,
                                              int hi, long long k, long long step) {
  const double lo_face = f[k];
  if (cell >= hi) return lo_face;
  return __dmul_rn(__dadd_rn(lo_face, f[k + step]), 0.5);  // = / 2 exactly
}
__device__ __forceinline__ St load_cell1(const StateP& u, const Grid& g, int i, int j) {
  const long long k = g.idx(i, j);
  St s{u.c[0][k], u.c[1][k], u.c[2][k], u.c[3][k], u.c[4][k], 0.0, 0.0, u.c[7][k]};
  s.bx = low_order_b(u.c[5], g, i, g.nx + g.ng - 1, k, 1);
  s.by = low_order_b(u.c[6], g, j, g.ny + g.ng - 1, k, g.pitch);
  return s;
}

// ---- face -> cell collocation (mhd_staggering.hpp:77-236) -----------------
__constant__ double c_f2c6[6] = {11, -93, 802, 802, -93, 11};
__constant__ double c_f2c8[8] = {-191, 1879, -9531, 68323, 68323, -9531, 1879, -191};
__constant__ double c_f2c4[4] = {-1, 13, 13, -1};
__constant__ double c_bary8[8] = {1, -7, 21, -35, 35, -21, 7, -1};
__constant__ double c_bary6[6] = {1, -5, 10, -10, 5, -1};
__constant__ double c_bary4[4] = {1, -3, 3, -1};
__constant__ double c_gx[4] = {0.0694318442029737124, 0.3300094782075718676,
                               0.6699905217924281324, 0.9305681557970262876};
__constant__ double c_gw[4] = {0.1739274225687269287, 0.3260725774312730713,
                               0.3260725774312730713, 0.1739274225687269287};

// Width-W collocation of the face samples f[k0 + step*q] for q = start..start+W-1
// at cell `cell` (W = 4, 6, 8 for 2, 3, 4 ghost layers).
template <int W>
__device__ double face_to_cell(const double* f, long long base, long long step, int cell,
                               int lo, int hi) {
  double cw[W];
#pragma unroll
  for (int k = 0; k < W; ++k) cw[k] = W == 8 ? c_f2c8[k] : W == 6 ? c_f2c6[k] : c_f2c4[k];
  const double den = W == 8 ? 120960.0 : W == 6 ? 1440.0 : 24.0;
  const int cs = cell - (W / 2 - 1);
  if (cs >= lo && cs + W - 1 <= hi) {
    double x[W];
#pragma unroll
    for (int k = 0; k < W; ++k) x[k] = __ldg(f + base + step * (long long)(cs + k));
    // Exact numerator rounded once, then one division (reference
    // scaled_rational_weighted_sum): a constant collocates to itself.
    return __ddiv_rn(exact_dot<W>(cw, x), den);
  }
  // One-sided outer-ghost closure: Gauss integral of the barycentric
  // interpolant through the W nearest faces (mhd_staggering.hpp:113-173).
  int start = cs < lo ? lo : cs;
  if (start + W - 1 > hi) start = hi - W + 1;
  double bw[W];
#pragma unroll
  for (int k = 0; k < W; ++k) bw[k] = W == 8 ? c_bary8[k] : W == 6 ? c_bary6[k] : c_bary4[k];
  const double rel = double(cell - start);
  double s = 0.0, c = 0.0;
  for (int q = 0; q < 4; ++q) {
    const double x = __dadd_rn(rel, c_gx[q]);
    double ds = 0.0, dc = 0.0;
    for (int k = 0; k < W; ++k) {
      double e;
      two_sum(ds, __ddiv_rn(bw[k], __dadd_rn(x, -double(k))), ds, e);
      dc = __dadd_rn(dc, e);
    }
    const double dsum = __dadd_rn(ds, dc);
    for (int k = 0; k < W; ++k) {
      const double wb = __dmul_rn(c_gw[q], bw[k]);
      const double v = f[base + step * (long long)(start + k)];
      const double t = __ddiv_rn(__ddiv_rn(__dmul_rn(wb, v), __dadd_rn(x, -double(k))), dsum);
      double e;
      two_sum(s, t, s, e);
      c = __dadd_rn(c, e);
    }
  }
  return __dadd_rn(s, c);
}

// ---- boundary closure (mhd_boundary_hip.hip:66-218) ------------------------
__device__ __forceinline__ void ghost_src(int n, int layer, bool lo, int mode, int& gi, int& si) {
  gi = lo ? -layer : n - 1 + layer;
  if (mode == 0) si = lo ? n - layer : layer - 1;
  else if (mode == 1) si = lo ? 0 : n - 1;
  else si = lo ? layer - 1 : n - layer;
}

// One ghost layer of one boundary line.  parts: bit 0 the fluid components
// (rho, momentum, energy, bz_cell; a wall flips the normal momentum), bit 1
// the staggered field (tangential face even; the normal face by its own rule).
__device__ __forceinline__ void fill_ghost(const Grid& g, const StateP& u, int axis, bool lo,
                                           int mode, int layer, int line, int parts) {
  const int n = axis == 0 ? g.nx : g.ny;
  int gi, si;
  ghost_src(n, layer, lo, mode, gi, si);
  auto at = [&](int a) { return axis == 0 ? g.idx(a, line) : g.idx(line, a); };
  const long long kd = at(gi), ks = at(si);
  const double sn = mode == 2 ? -1.0 : 1.0;
  if (parts & 1) {
    u.c[0][kd] = u.c[0][ks];
    u.c[1][kd] = (axis == 0 ? sn : 1.0) * u.c[1][ks];
    u.c[2][kd] = (axis == 1 ? sn : 1.0) * u.c[2][ks];
    u.c[3][kd] = u.c[3][ks];
    u.c[4][kd] = u.c[4][ks];
    u.c[7][kd] = u.c[7][ks];
  }
  if (!(parts & 2)) return;
  double* bn = axis == 0 ? u.c[5] : u.c[6];
  double* bt = axis == 0 ? u.c[6] : u.c[5];
  bt[kd] = bt[ks];
  if (mode == 2) {
    if (lo) {
      bn[at(0)] = 0.0;
      bn[at(-layer)] = -bn[at(layer)];
    } else if (layer == 1) {
      bn[at(n)] = 0.0;
    } else {
      bn[at(n + layer - 1)] = -bn[at(n - (layer - 1))];
    }
  } else if (mode == 1 && !lo) {
    // the physical high face n is evolved by CT; only faces beyond it copy it
    if (layer > 1) bn[at(n - 1 + layer)] = bn[at(n)];
  } else {
    bn[kd] = sn * bn[ks];
  }
}

// axis 0: the x sides (both), all padded rows; axis 1: the y sides over all
// padded columns (run after axis 0 so the corner blocks close last).
__device__ __forceinline__ void b_fill_ghosts(const Grid& g, const StateP& u, int axis, int bx) {
  const int lines = (axis == 0 ? g.ny : g.nx) + 2 * g.ng;
  const int t = bx * blockDim.x + threadIdx.x;
  if (t >= 2 * g.ng * lines) return;
  const int side = t / (g.ng * lines);
  const int rem = t - side * g.ng * lines;
  fill_ghost(g, u, axis, side == 0, g.bc[axis * 2 + side], rem / lines + 1, rem % lines - g.ng, 3);
}

__global__ void k_fill_ghosts(Grid g, StateP u, int axis) {
  b_fill_ghosts(g, u, axis, blockIdx.x);
}

// ---- admissible convex fraction (mhd_reduce.hip:120-209) ------------------
__device__ __forceinline__ double convex_q(const St& a, const St& b, double th) {
  const double omt = 1.0 - th;
  const double rho = omt * a.rho + th * b.rho;
  if (!(rho > 0.0) || !isfinite(rho)) return -kInf;
  const double mx = omt * a.mx + th * b.mx, my = omt * a.my + th * b.my;
  const double mz = omt * a.mz + th * b.mz, e = omt * a.E + th * b.E;
  const double bx = omt * a.bx + th * b.bx, by = omt * a.by + th * b.by;
  const double bz = omt * a.bz + th * b.bz;
  const double q = (e - kin_mom(mx, my, mz, rho)) - half_sq3(bx, by, bz);
  return isfinite(q) ? q : -kInf;
}
// Internal energy certainly positive: plain arithmetic with a margin far
// above its rounding error (a few ulps of E + kinetic + magnetic), so the
// sign agrees with the reference's scaled form whenever this returns true.
__device__ __forceinline__ bool surely_admissible(const St& s) {
  if (!(isfinite(s.rho) && s.rho > 0.0 && isfinite(s.mx) && isfinite(s.my) && isfinite(s.mz) &&
        isfinite(s.E) && isfinite(s.bx) && isfinite(s.by) && isfinite(s.bz)))
    return false;
  const double kin = 0.5 * ((s.mx * s.mx + s.my * s.my + s.mz * s.mz) / s.rho);
  const double mag = 0.5 * (s.bx * s.bx + s.by * s.by + s.bz * s.bz);
  const double q = (s.E - kin) - mag;
  return isfinite(q) && q > 1e-12 * (fabs(s.E) + kin + mag);
}

__device__ double admissible_fraction(const St& a, const St& b) {
  // both end points certainly admissible: the exact path returns 1 as well
  // (convex_q at theta 0 and 1 are the end points themselves)
  if (surely_admissible(a) && surely_admissible(b)) return 1.0;
  const double qa = convex_q(a, b, 0.0);
  if (!(a.rho > 0.0) || !(qa > 0.0) || !isfinite(a.rho) || !isfinite(qa)) return 0.0;
  if (!(isfinite(b.rho) && isfinite(b.mx) && isfinite(b.my) && isfinite(b.mz) &&
        isfinite(b.E) && isfinite(b.bx) && isfinite(b.by) && isfinite(b.bz)))
    return 0.0;
  double hi = 1.0;
  if (b.rho <= 0.0) {
    const double den = a.rho - b.rho;
    hi = den > 0.0 ? a.rho / den : 0.0;
    hi = fmin(fmax(hi, 0.0), 1.0);
  }
  if (convex_q(a, b, hi) > 0.0) return hi;
  double lo = 0.0;
  for (int it = 0; it < 56; ++it) {
    const double mid = 0.5 * (lo + hi);
    if (convex_q(a, b, mid) > 0.0) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}

// atomicMax of non-negative double bit patterns, one atomic per group of
// converged lanes: the per-cell maxima of a developed flow hit one address
// from nearly every cell, and same-address atomics serialise in L2.  The max
// is exact and order-free, so the stored value is the per-cell one's.
__device__ __forceinline__ void atomic_max_lanes(unsigned long long* dst, unsigned long long v) {
  const cg::coalesced_group grp = cg::coalesced_threads();
  const unsigned long long m = cg::reduce(grp, v, cg::greater<unsigned long long>());
  if (grp.thread_rank() == 0 && m != 0ull) atomicMax(dst, m);
}

// ulp of a finite double as used by the solenoidality preflight
// (numerics/mhd_background_metrics.hpp:105-121).
__device__ __forceinline__ double ulp_of(double x) {
  const double m = fabs(x);
  if (!isfinite(x)) return kInf;
  if (m < kTiny) return 4.9406564584124654e-324;
  int e;
  frexp(m, &e);
  return ldexp(0.5, e - 52);
}

// Discrete div B of interior cell k relative to the directional scale
// (mhd_reduce.hip:556-700, solver mhd_solver.cpp:1196-1222): the residual
// the rounding envelope does not explain and the scale |d1| + |d2|, as bit
// patterns of non-negative doubles (0 = nothing to record; a non-finite
// stencil records an infinite residual).
__device__ __forceinline__ void divb_cell(const Grid& g, const StateP& u, long long k,
                                          int solver_owned, unsigned long long& rb,
                                          unsigned long long& sb) {
  const double bxl = u.c[5][k], bxh = u.c[5][k + 1];
  const double byl = u.c[6][k], byh = u.c[6][k + g.pitch];
  const double rdx = pow2_recip(g.dx), rdy = pow2_recip(g.dy);
  const double d1 = div_by(__dadd_rn(bxh, -bxl), g.dx, rdx);
  const double d2 = div_by(__dadd_rn(byh, -byl), g.dy, rdy);
  const double res = __dadd_rn(d1, d2);
  const double scale = __dadd_rn(fabs(d1), fabs(d2));
  const double unc = __dadd_rn(div_by(__dadd_rn(ulp_of(bxh), ulp_of(bxl)), g.dx, rdx),
                               div_by(__dadd_rn(ulp_of(byh), ulp_of(byl)), g.dy, rdy));
  bool explained;
  if (solver_owned) {
    explained = fabs(res) <= 1024.0 * unc;
  } else {
    explained = d1 != 0.0 && d2 != 0.0 && (signbit(d1) != signbit(d2)) &&
                fabs(res) <= 0.5 * scale && fabs(res) <= 1024.0 * unc;
  }
  const double r = explained ? 0.0 : fabs(res);
  const bool finite = isfinite(r) && isfinite(scale);
  rb = !finite ? dbits(kInf) : r > 0.0 ? dbits(r) : 0ull;
  sb = finite && scale > 0.0 ? dbits(scale) : 0ull;
}

// Collocate the candidate state's in-plane field (padded range) and, for
// interior cells, run the admissibility fraction against `base` and the
// live-state preflights.  theta_mask: bit0 collocation order 0, bit1 order 1,
// bit2 order 1 only when the live state's low-order anchor is admissible.
template <int W>
__device__ __forceinline__ void b_colloc_check(const Grid& g, const StateP& cand, const StateP& base, int has_base,
                                               int theta_mask, int live_checks, int solver_owned,
                                               double gamma, Ctl* ctl, int bx, int by) {
  const int i = bx * blockDim.x + threadIdx.x - g.ng;
  const int j = by * blockDim.y + threadIdx.y - g.ng;
  if (i >= g.nx + g.ng || j >= g.ny + g.ng) return;
  if (ctl->status & ~kStatusDone) return;
  const long long k = g.idx(i, j);
  const double bxc = face_to_cell<W>(cand.c[5], (long long)g.idx(0, j) - 0, 1, i, -g.ng,
                                     g.nx + g.ng - 1);
  const double byc = face_to_cell<W>(cand.c[6], (long long)g.idx(i, 0), g.pitch, j, -g.ng,
                                     g.ny + g.ng - 1);
  cand.bxc[k] = bxc;
  cand.byc[k] = byc;
  if (i < 0 || j < 0 || i >= g.nx || j >= g.ny || !g.in_window(i, j)) return;
  const St b{cand.c[0][k], cand.c[1][k], cand.c[2][k], cand.c[3][k], cand.c[4][k], bxc, byc,
             cand.c[7][k]};
  if (has_base) {
    double th = 1.0;
    if (theta_mask & 1) {
      const St a{base.c[0][k], base.c[1][k], base.c[2][k], base.c[3][k], base.c[4][k],
                 base.bxc[k], base.byc[k], base.c[7][k]};
      th = fmin(th, admissible_fraction(a, b));
    }
    const bool anchor = (theta_mask & 4) && ctl->anchor_ok != 0;
    if ((theta_mask & 2) || anchor) {
      th = fmin(th, admissible_fraction(load_cell1(base, g, i, j), load_cell1(cand, g, i, j)));
    }
    if (!(th >= 1.0)) {
      atomicMin(&ctl->theta, dbits(isfinite(th) ? th : 0.0));
      atomicOr(&ctl->status, kStatusRetry);
    }
  }
  if (live_checks) {
    const double t0 = admissible_fraction(b, b);
    if (!(t0 >= 1.0)) atomicMin(&ctl->live_theta, dbits(t0));
    const St b1 = load_cell1(cand, g, i, j);
    const double t1 = admissible_fraction(b1, b1);
    if (!(t1 >= 1.0)) atomicMin(&ctl->anchor_theta, dbits(t1));
    unsigned long long rb, sb;
    divb_cell(g, cand, k, solver_owned, rb, sb);
    atomic_max_lanes(&ctl->divb_res, rb);
    atomic_max_lanes(&ctl->divb_scale, sb);
  }
}

// Three blocks per SM: the bisection and ulp paths that are rarely taken spill
// at 80 registers, and the common path runs 22% faster than at 122 registers.
template <int W>
__global__ void __launch_bounds__(256, 3)
    k_colloc_check(Grid g, StateP cand, StateP base, int has_base, int theta_mask,
                   int live_checks, int solver_owned, double gamma, Ctl* ctl) {
  b_colloc_check<W>(g, cand, base, has_base, theta_mask, live_checks, solver_owned, gamma, ctl, blockIdx.x,
                    blockIdx.y);
}

}  // namespace

// ===========================================================================
// Reconstruction (reference mhd_reconstruct.hip:150-670)
// ===========================================================================
namespace {

template <int DIR>
__device__ __forceinline__ St rot(const St& s) {
  return DIR == 0 ? s : swap_xy(s);
}

// Replace the reconstructed normal field by the shared CT face value while
// keeping the gas pressure (mhd_reconstruct.hip:150-161).  The compensated
// sum returns E bit for bit when the two values agree.
template <int DIR>
__device__ __forceinline__ void set_normal_b(St& s, double v) {
  double& bn = DIR == 0 ? s.bx : s.by;
  s.E = crsum3(s.E, __dmul_rn(v, 0.5 * v), __dmul_rn(bn, -0.5 * bn));
  bn = v;
}

// ---- characteristic eigensystem, one wave at a time ----------------------
// Scalars of the eigensystem about a canonical (x-normal) state
// (mhd_eigensystem.hpp:63-171), shared by all seven waves.
struct Eg {
  double rho, sr, cf, cs, a, af, as, b1, b2, sbn, vn, vt1, vt2, bt1, bt2;
  double ia2, ra2, gm1, hv2, ir, igm;
  bool sure;  // L R = I within the tolerance for certain (below)
};
constexpr double kRs2 = 0.7071067811865475;  // 1/sqrt(2) rounded

// The magnetosonic speeds and the fast / slow normalisations keep the
// reference's scaled forms and uncontracted products: where the transverse
// field vanishes, af^2 is a difference of nearly equal squares and af its
// square root, so a one-ulp change of any input moves af by ~1e-8 and the
// face states by ~1e-11.  Quantities that feed only the eigenvector
// entries (velocities, transverse unit vector, 1/a^2, |v|^2/2) share one
// reciprocal each instead of a division per term (a rounding-level
// difference).
template <class D>
__device__ __forceinline__ Eg eig_scalars_by(D& dv, const St& s, double gamma) {
  Eg e;
  e.rho = s.rho;
  e.sr = sqrt(e.rho);
  const auto dsr = dv.by(e.sr);
  const double ir = 1.0 / s.rho;
  const Pr w{s.rho, s.mx * ir, s.my * ir, s.mz * ir, pressure(dv, dsr, s, gamma), s.bx, s.by, s.bz};
  const double p = w.p > 0.0 ? w.p : 0.0;
  e.bt1 = w.by;
  e.bt2 = w.bz;
  double cax, ca, den, clip = 0.0;
  magnetosonic(dv, dsr, p, w.bx, w.by, w.bz, gamma, e.cf, e.cs, e.a, cax, ca);
  {
    const auto sc = dv.by(e.cf > 0.0 ? e.cf : 1.0);
    const double cfn = sc.of(e.cf), csn = sc.of(e.cs), an = sc.of(e.a);
    den = sub(mul(cfn, cfn), mul(csn, csn));
    if (den <= mul(64.0 * kEps, add(mul(cfn, cfn), mul(csn, csn)))) {
      e.af = kRs2;
      e.as = kRs2;
      den = 0.0;
    } else {
      const auto dd = dv.by(den);
      const double af2 = dd.of(sub(mul(an, an), mul(csn, csn)));
      const double as2 = dd.of(sub(mul(cfn, cfn), mul(an, an)));
      e.af = sqrt(af2 < 0.0 ? 0.0 : af2);
      e.as = sqrt(as2 < 0.0 ? 0.0 : as2);
      const double least = af2 < as2 ? af2 : as2;
      clip = least < 0.0 ? -least : 0.0;
    }
  }
  {
    const double bt = scaled_norm3(dv, w.by, w.bz, 0.0);
    const double fs = e.a > ca ? e.a : ca;
    if (bt == 0.0 || dsr.of(bt) <= 64.0 * kEps * (fs + kTiny)) {
      e.b1 = kRs2;
      e.b2 = kRs2;
    } else {
      const double ibt = 1.0 / bt;
      e.b1 = w.by * ibt;
      e.b2 = w.bz * ibt;
    }
  }
  e.sbn = w.bx >= 0.0 ? 1.0 : -1.0;
  e.vn = w.vx;
  e.vt1 = w.vy;
  e.vt2 = w.vz;
  const double ia = e.a > 0.0 ? 1.0 / e.a : 0.0;
  e.ia2 = ia * ia;
  e.ra2 = gamma * p;
  e.gm1 = gamma - 1.0;
  e.hv2 = 0.5 * ((e.vn * e.vn + e.vt1 * e.vt1) + e.vt2 * e.vt2);
  e.ir = ir;
  e.igm = 1.0 / e.gm1;
  // A bound that shows the L R = I check to pass without forming it.  With
  // k = c_f / a, M = (|v_n| + |v_t1| + |v_t2|) / a, b = (|B_t1| + |B_t2|) /
  // (a sqrt(rho)), g = gamma - 1 and d = 1 - c_s^2 / c_f^2, every sum of
  // magnitudes sum_m |L_im R_mj| is at most
  //   S = max(rho, 1/rho) max(a, 1/a) F,
  //   F = 3 + 3 k + 2 M + 1.5 k^2 + (1 + 4 g) k M + 2 g M^2 + 3 g b
  // (term by term over the fast, slow, Alfven and entropy rows and columns).
  // The rounding of the entries (at most six operations each side) and of the
  // product is below 24 u S, u = eps / 2, in any order of summation.  The
  // rounding of the normalisations moves af^2 + as^2 - 1, and with the factor
  // k^2 the sum af^2 c_f^2 + as^2 c_s^2 = a^2, by less than 19 u / d, and a
  // negative square set to zero by its size c (where c_f or c_s itself is off
  // by rounding): together below 24 u k^2 (1 / d + c / (24 u)).  So S + k^2
  // (1 / d + c / (24 u)) <= 80 keeps all of it, with 20 u for the constants,
  // below 2048 u = 1024 eps.  Most faces of a flow near Mach one pass it; the
  // others (strong scales, near-degenerate fans, high Mach numbers) take the
  // check itself.  Reconstruction 7.6 -> 6.4 ms per step on a flow at 2048^2
  // MP7, with the shared-memory strides of mp_faces_warp.
  {
    const double k = e.cf * ia, g = e.gm1;
    const double M = (fabs(e.vn) + fabs(e.vt1) + fabs(e.vt2)) * ia;
    const double b = (fabs(e.bt1) + fabs(e.bt2)) * (ia * e.sr * ir);
    const double F = 3.0 + 3.0 * (k + g * b) + 1.5 * (k * k) + M * (2.0 + (1.0 + 4.0 * g) * k + 2.0 * g * M);
    const double W = (e.rho > ir ? e.rho : ir) * (e.a > ia ? e.a : ia);
    e.sure = (80.0 - W * F) * den >= k * k * fma(den * clip, 3.8e14, 1.0);
  }
  return e;
}

__device__ __noinline__ Eg eig_scalars_plain(const St& s, double gamma) {
  PlainDiv d;
  return eig_scalars_by(d, s, gamma);
}
// The eigen scalars are a quarter of the reconstruction's instructions and one
// long dependent chain, most of it 26 divisions by twelve divisors; sharing
// each divisor's reciprocal keeps the bits (flow 2048^2 MP7 reconstruction
// 6.29 -> 5.86 ms per step, rotor 4096^2 26.0 -> 23.0).  Divisors outside the
// shared form's range are tested once at the end: a select per quotient
// measured slower than the divisions.
__device__ __forceinline__ Eg eig_scalars(const St& s, double gamma) {
  SharedDiv d;
  const Eg e = eig_scalars_by(d, s, gamma);
  return d.bad ? eig_scalars_plain(s, gamma) : e;
}

// Primitive left row and right column of wave k (mhd_eigensystem.hpp:176-320);
// k = 7 (the spare lane) gets zeros.
__device__ __forceinline__ void wave_vectors(const Eg& e, int k, double* lp, double* rp) {
#pragma unroll
  for (int v = 0; v < 7; ++v) {
    lp[v] = 0.0;
    rp[v] = 0.0;
  }
  const double rho = e.rho;
  const double qf = e.cf * e.af * e.sbn, qs = e.cs * e.as * e.sbn;
  const double Af = e.a * e.af * e.sr, As = e.a * e.as * e.sr;
  const double Nf = 0.5 * e.ia2, s2 = kRs2;
  if (k == 0 || k == 6) {
    rp[0] = rho * e.af;
    rp[1] = k == 0 ? -e.af * e.cf : e.af * e.cf;
    rp[2] = k == 0 ? qs * e.b1 : -qs * e.b1;
    rp[3] = k == 0 ? qs * e.b2 : -qs * e.b2;
    rp[4] = e.af * e.ra2;
    rp[5] = As * e.b1;
    rp[6] = As * e.b2;
    lp[1] = k == 0 ? -Nf * e.af * e.cf : Nf * e.af * e.cf;
    lp[2] = k == 0 ? Nf * qs * e.b1 : -Nf * qs * e.b1;
    lp[3] = k == 0 ? Nf * qs * e.b2 : -Nf * qs * e.b2;
    lp[4] = Nf * e.af * e.ir;
    lp[5] = Nf * As * e.b1 * e.ir;
    lp[6] = Nf * As * e.b2 * e.ir;
  } else if (k == 1 || k == 5) {
    rp[2] = -e.b2 * s2;
    rp[3] = e.b1 * s2;
    rp[5] = k == 1 ? -e.sbn * e.b2 * s2 * e.sr : e.sbn * e.b2 * s2 * e.sr;
    rp[6] = k == 1 ? e.sbn * e.b1 * s2 * e.sr : -e.sbn * e.b1 * s2 * e.sr;
    lp[2] = -e.b2 * s2;
    lp[3] = e.b1 * s2;
    const double isr = e.sr * e.ir;
    lp[5] = k == 1 ? -e.sbn * e.b2 * s2 * isr : e.sbn * e.b2 * s2 * isr;
    lp[6] = k == 1 ? e.sbn * e.b1 * s2 * isr : -e.sbn * e.b1 * s2 * isr;
  } else if (k == 2 || k == 4) {
    rp[0] = rho * e.as;
    rp[1] = k == 2 ? -e.as * e.cs : e.as * e.cs;
    rp[2] = k == 2 ? -qf * e.b1 : qf * e.b1;
    rp[3] = k == 2 ? -qf * e.b2 : qf * e.b2;
    rp[4] = e.as * e.ra2;
    rp[5] = -Af * e.b1;
    rp[6] = -Af * e.b2;
    lp[1] = k == 2 ? -Nf * e.as * e.cs : Nf * e.as * e.cs;
    lp[2] = k == 2 ? -Nf * qf * e.b1 : Nf * qf * e.b1;
    lp[3] = k == 2 ? -Nf * qf * e.b2 : Nf * qf * e.b2;
    lp[4] = Nf * e.as * e.ir;
    lp[5] = -Nf * Af * e.b1 * e.ir;
    lp[6] = -Nf * Af * e.b2 * e.ir;
  } else if (k == 3) {
    rp[0] = 1.0;
    lp[0] = 1.0;
    lp[4] = -e.ia2;
  }
}

// One thread per face, wave loop rolled: L row and R column of each wave are
// rebuilt from the shared eigen scalars when needed, so only the stencil
// deltas stay resident.  Same arithmetic per entry as build_eig.
__device__ __forceinline__ void conserved_row_col(const Eg& e, int k, double* Lr, double* Rc) {
  double lp[7], rp[7];
  wave_vectors(e, k, lp, rp);
  const double gv = e.gm1;
  Lr[0] = (((lp[0] * 1.0 + lp[1] * (-e.vn * e.ir)) + lp[2] * (-e.vt1 * e.ir)) +
           lp[3] * (-e.vt2 * e.ir)) + lp[4] * (gv * e.hv2);
  Lr[1] = lp[1] * e.ir + lp[4] * (-gv * e.vn);
  Lr[2] = lp[2] * e.ir + lp[4] * (-gv * e.vt1);
  Lr[3] = lp[3] * e.ir + lp[4] * (-gv * e.vt2);
  Lr[4] = lp[4] * gv;
  Lr[5] = lp[4] * (-gv * e.bt1) + lp[5];
  Lr[6] = lp[4] * (-gv * e.bt2) + lp[6];
  Rc[0] = rp[0];
  Rc[1] = e.vn * rp[0] + e.rho * rp[1];
  Rc[2] = e.vt1 * rp[0] + e.rho * rp[2];
  Rc[3] = e.vt2 * rp[0] + e.rho * rp[3];
  Rc[4] = (((((e.hv2 * rp[0] + (e.rho * e.vn) * rp[1]) + (e.rho * e.vt1) * rp[2]) +
             (e.rho * e.vt2) * rp[3]) + e.igm * rp[4]) + e.bt1 * rp[5]) + e.bt2 * rp[6];
  Rc[5] = rp[5];
  Rc[6] = rp[6];
}

// Dynamic shared memory of every kernel that runs mp_pair_loop: 98 doubles
// (7 L rows + 7 R columns) per thread of a 128-thread block.
constexpr int kReconThreads = 128;
constexpr size_t kReconSmem = 98 * kReconThreads * sizeof(double);

template <int DIR, int H>
__device__ void mp_pair_loop(const StateP& u, long long k0, long long step, double gamma, St& ul,
                             St& ur, bool* fired_l = nullptr, bool* fired_r = nullptr) {
  constexpr int S = 2 * H + 2, W = 2 * H + 1;
  const St cl = load_cell(u, k0 - step), cr = load_cell(u, k0);
  St ref;
  ref.rho = 0.5 * cl.rho + 0.5 * cr.rho;
  ref.mx = 0.5 * cl.mx + 0.5 * cr.mx;
  ref.my = 0.5 * cl.my + 0.5 * cr.my;
  ref.mz = 0.5 * cl.mz + 0.5 * cr.mz;
  ref.E = 0.5 * cl.E + 0.5 * cr.E;
  ref.bx = 0.5 * cl.bx + 0.5 * cr.bx;
  ref.by = 0.5 * cl.by + 0.5 * cr.by;
  ref.bz = 0.5 * cl.bz + 0.5 * cr.bz;
  const St c = rot<DIR>(ref);
  const Eg e = eig_scalars(c, gamma);
  // All seven L rows and R columns built once into this thread's slots of
  // dynamic shared memory (kReconSmemDoubles per thread, stride = threads per
  // block), then the L R = I check (mhd_eigensystem.hpp:416-430) with R
  // resident in two halves (4 + 3).  |d| <= 1024 eps is tested as
  // d^2 <= (1024 eps)^2, the same decision since 1024 eps is a power of two
  // (and false for NaN and infinity).
  extern __shared__ double dsm[];
  const int ST = blockDim.x * blockDim.y;
  double* LR = dsm + (threadIdx.y * blockDim.x + threadIdx.x);
#pragma unroll 1
  for (int k = 0; k < 7; ++k) {
    double Lr[7], Rc[7];
    conserved_row_col(e, k, Lr, Rc);
#pragma unroll
    for (int m = 0; m < 7; ++m) {
      LR[(k * 7 + m) * ST] = Lr[m];
      LR[(49 + k * 7 + m) * ST] = Rc[m];
    }
  }
  bool usable = true;
  constexpr double kT2 = (1024.0 * kEps) * (1024.0 * kEps);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    constexpr int kCols = 4;
    const int j0 = half * kCols, nj = half == 0 ? kCols : 7 - kCols;
    double Rm[kCols][7];
#pragma unroll
    for (int jj = 0; jj < kCols; ++jj)
#pragma unroll
      for (int m = 0; m < 7; ++m) Rm[jj][m] = jj < nj ? LR[(49 + (j0 + jj) * 7 + m) * ST] : 0.0;
#pragma unroll 1
    for (int i = 0; i < 7; ++i) {
      double Lr[7];
#pragma unroll
      for (int m = 0; m < 7; ++m) Lr[m] = LR[(i * 7 + m) * ST];
#pragma unroll
      for (int jj = 0; jj < kCols; ++jj) {
        if (jj >= nj) continue;
        double dot = 0.0;
#pragma unroll
        for (int m = 0; m < 7; ++m) dot += Lr[m] * Rm[jj][m];
        const double d = dot - (i == j0 + jj ? 1.0 : 0.0);
        usable = usable && (d * d <= kT2);
      }
    }
  }
  // stencil deltas in the canonical frame
  double u7[S][7];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const St d = rot<DIR>(load_cell(u, k0 + (long long)(s - 1 - H) * step));
    u7[s][0] = d.rho - c.rho;
    u7[s][1] = d.mx - c.mx;
    u7[s][2] = d.my - c.my;
    u7[s][3] = d.mz - c.mz;
    u7[s][4] = d.E - c.E;
    u7[s][5] = d.by - c.by;
    u7[s][6] = d.bz - c.bz;
  }
  double dl[7], dr[7];
#pragma unroll
  for (int v = 0; v < 7; ++v) {
    dl[v] = 0.0;
    dr[v] = 0.0;
  }
#pragma unroll 1
  for (int k = 0; k < 7; ++k) {
    double Lr[7];
    if (usable) {
#pragma unroll
      for (int m = 0; m < 7; ++m) Lr[m] = LR[(k * 7 + m) * ST];
    } else {
#pragma unroll
      for (int v = 0; v < 7; ++v) Lr[v] = v == k ? 1.0 : 0.0;
    }
    double ch[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      double acc = 0.0;
#pragma unroll
      for (int v = 0; v < 7; ++v) acc += Lr[v] * u7[s][v];
      ch[s] = acc;
    }
    double win[W];
    bool f;
#pragma unroll
    for (int s = 0; s < W; ++s) win[s] = ch[s];
    const double wl = mp_recon<W>(win, f);
    if (fired_l && f) *fired_l = true;
#pragma unroll
    for (int s = 0; s < W; ++s) win[s] = ch[W - s];
    const double wr = mp_recon<W>(win, f);
    if (fired_r && f) *fired_r = true;
    double Rc[7];
    if (usable) {
#pragma unroll
      for (int m = 0; m < 7; ++m) Rc[m] = LR[(49 + k * 7 + m) * ST];
    } else {
#pragma unroll
      for (int v = 0; v < 7; ++v) Rc[v] = v == k ? 1.0 : 0.0;
    }
#pragma unroll
    for (int v = 0; v < 7; ++v) {
      dl[v] += Rc[v] * wl;
      dr[v] += Rc[v] * wr;
    }
  }
  const St sl{c.rho + dl[0], c.mx + dl[1], c.my + dl[2], c.mz + dl[3],
              c.E + dl[4],   c.bx,         c.by + dl[5], c.bz + dl[6]};
  const St sr{c.rho + dr[0], c.mx + dr[1], c.my + dr[2], c.mz + dr[3],
              c.E + dr[4],   c.bx,         c.by + dr[5], c.bz + dr[6]};
  ul = rot<DIR>(sl);
  ur = rot<DIR>(sr);
}

// Component-wise unlimited MP interpolation of the same conserved deltas:
// the characteristic path with L = R = I and no limiter, which equals the
// characteristic result wherever the limiter accepts every wave (R L = I).
// The components are independent, so each is loaded, interpolated and
// finished before the next (few live registers); the sums are those of the
// whole-state form.
template <int DIR, int H>
__device__ void mp_pair_lin(const StateP& u, long long k0, long long step, St& ul, St& ur) {
  constexpr int S = 2 * H + 2, W = 2 * H + 1;
  double dl[8], dr[8], cv[8];
  // canonical frame: rho, m_n, m_t1, m_t2, E, b_n, b_t1, b_t2
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const double* a = v == 0 ? u.c[0]
                      : v == 1 ? (DIR == 0 ? u.c[1] : u.c[2])
                      : v == 2 ? (DIR == 0 ? u.c[2] : u.c[1])
                      : v == 3 ? u.c[3]
                      : v == 4 ? u.c[4]
                      : v == 5 ? (DIR == 0 ? u.bxc : u.byc)
                      : v == 6 ? (DIR == 0 ? u.byc : u.bxc)
                               : u.c[7];
    const double c = 0.5 * __ldg(a + k0 - step) + 0.5 * __ldg(a + k0);
    cv[v] = c;
    if (v == 5) continue;  // the normal field is not reconstructed
    double w[S];
#pragma unroll
    for (int t = 0; t < S; ++t) w[t] = __ldg(a + k0 + (long long)(t - 1 - H) * step) - c;
    dl[v] = mp_interp_plain<W>(w);
    double wr[W];
#pragma unroll
    for (int t = 0; t < W; ++t) wr[t] = w[W - t];
    dr[v] = mp_interp_plain<W>(wr);
  }
  const St sl{cv[0] + dl[0], cv[1] + dl[1], cv[2] + dl[2], cv[3] + dl[3],
              cv[4] + dl[4], cv[5],         cv[6] + dl[6], cv[7] + dl[7]};
  const St sr{cv[0] + dr[0], cv[1] + dr[1], cv[2] + dr[2], cv[3] + dr[3],
              cv[4] + dr[4], cv[5],         cv[6] + dr[6], cv[7] + dr[7]};
  ul = rot<DIR>(sl);
  ur = rot<DIR>(sr);
}

template <int DIR, int ORDER, int MODE>
__device__ __forceinline__ void finish_face(const Grid& g, const StateP& u, const IfaceP& out,
                                            double gamma, int i, int j, long long k0,
                                            long long step, St ul, St ur);

// ---- warp-cooperative characteristic MP reconstruction --------------------
// The characteristic path of mp_pair_loop with the work of one face spread
// over four lanes, lane r holding the pair of waves r and 6 - r (lane 3 the
// entropy wave alone), so that a thread carries two waves' L rows and
// projected stencils instead of all seven, and has two independent chains.
// A warp owns 32 faces:
//   phase 1  lane = face: reference state and eigen scalars -> shared memory
//   phase 2  4 rounds of 8 faces, lane = (face, wave pair): L rows and R
//            columns, the L R = I check (R columns exchanged through shared
//            memory), the stencil deltas (lane = two stencil cells),
//            projection, MP limiter on both sides, back-projection (lane =
//            components r and r + 4)
//   phase 3  lane = face: states, fallback chain, stores (finish_face)
// The pair's rows and columns are kept as their thermal / magnetic and
// velocity parts (WavePair) and both face states of a wave come from one
// limiter evaluation (mp_pair_limit): 225 -> 177 warp instructions a face,
// 433 -> 326 us per 1024^2 MP7 launch.  The two paths agree to rounding.  Four
// lanes per face (not seven) because the exchanged operands are read once
// per lane: each shared-memory load costs one wavefront per half-warp whether
// or not the lanes share its address.
//
// Per-warp shared memory (doubles): a face record [kRec] rows of kRecS, and
// eight group buffers.  A group holds the four pairs' columns, 12 doubles
// apart (T components 0-6, V components 1-4 at offset 8), then the stencil
// deltas [8][7], whose first 16 slots later hold the face values (left 0-6,
// right 8-14).  The strides keep the exchange off common banks: 16-byte column
// stores at 12 r + 100 g, delta stores at 7 c + 100 g and the transposed
// back-projection stores at 36 v + f are conflict-free or two-way (with 8, 114
// and 32 the stores took 184 wavefronts a round against 92, and the L1 data
// pipe, the kernel's tightest resource, was 72% busy).
constexpr int kRecC = 0;    // canonical reference state, 8 components
constexpr int kRecE = 8;    // 16 eigen scalars, later dl[7] and dr[7]
constexpr int kRec = 24, kRecS = 36;
constexpr int kPair = 12, kPairV = 8, kGrpD = 44, kGrpW = 44, kGrpDoubles = 100;
constexpr int kGroups = 8;
constexpr int kWarpReconDoubles = kRec * kRecS + kGroups * kGrpDoubles;
constexpr int kReconWarps = 4;
constexpr size_t kReconWarpSmem = size_t(kReconWarps) * kWarpReconDoubles * sizeof(double);

// The pair of waves r and 6 - r (r = 0 fast, 1 Alfven, 2 slow; r = 3 the
// entropy wave alone) as its thermal / magnetic part and its velocity part:
// the rows are L_r = T - V and L_(6-r) = T + V, the columns likewise (the
// Alfven wave 1 with its overall sign reversed, which cancels between row and
// column and leaves the limiter's odd function unchanged).  Entries as in
// wave_vectors and conserved_row_col; V touches the momenta (and, in a row,
// the density, in a column the energy) only.  Alfven vectors are the
// magnetosonic ones with the transverse direction turned by 90 degrees.
struct WavePair {
  double lt[7], lv[4];  // row parts; lv: components 0-3
  double rt[7], rv[4];  // column parts; rv: components 1-4
};
__device__ __forceinline__ void wave_pair(const Eg& e, int r, WavePair& w) {
  const bool fast = r == 0, alf = r == 1, ent = r == 3, ms = !alf && !ent;
  const double al = fast ? e.af : e.as, cc = fast ? e.cf : e.cs;
  const double ax = fast ? e.as : e.af, cx = fast ? e.cs : e.cf;
  const double sx = fast ? -e.sbn : e.sbn, Nf = 0.5 * e.ia2;
  const double t1 = alf ? -e.b2 : e.b1, t2 = alf ? e.b1 : e.b2;
  // transverse velocity and field amplitudes
  const double qv = ms ? cx * ax * sx : (alf ? kRs2 : 0.0);
  const double qb = ms ? (fast ? ax : -ax) * e.a * e.sr : (alf ? -e.sbn * kRs2 * e.sr : 0.0);
  const double vn = ms ? al * cc : 0.0, v1 = qv * t1, v2 = qv * t2;
  const double r0 = ms ? e.rho * al : (ent ? 1.0 : 0.0), rp = ms ? al * e.ra2 : 0.0;
  const double r5 = qb * t1, r6 = qb * t2;
  const double fl = (ms ? Nf : 1.0) * e.ir;
  const double l1 = fl * vn, l2 = fl * v1, l3 = fl * v2;
  w.lv[0] = -(l1 * e.vn + l2 * e.vt1 + l3 * e.vt2);
  w.lv[1] = l1;
  w.lv[2] = l2;
  w.lv[3] = l3;
  const double g = (ms ? fl * al : (ent ? -e.ia2 : 0.0)) * e.gm1;
  w.lt[0] = g * e.hv2 + (ent ? 1.0 : 0.0);
  w.lt[1] = -g * e.vn;
  w.lt[2] = -g * e.vt1;
  w.lt[3] = -g * e.vt2;
  w.lt[4] = g;
  w.lt[5] = fl * r5 - g * e.bt1;
  w.lt[6] = fl * r6 - g * e.bt2;
  w.rv[0] = e.rho * vn;
  w.rv[1] = e.rho * v1;
  w.rv[2] = e.rho * v2;
  w.rv[3] = e.vn * w.rv[0] + e.vt1 * w.rv[1] + e.vt2 * w.rv[2];
  w.rt[0] = r0;
  w.rt[1] = e.vn * r0;
  w.rt[2] = e.vt1 * r0;
  w.rt[3] = e.vt2 * r0;
  w.rt[4] = (e.hv2 * r0 + e.igm * rp) + (e.bt1 * r5 + e.bt2 * r6);
  w.rt[5] = r5;
  w.rt[6] = r6;
}

// The reconstructed components (rho, m_n, m_t1, m_t2, E, B_t1, B_t2) of a cell.
template <int DIR>
__device__ __forceinline__ void cell7(const StateP& u, long long k, double* v) {
  v[0] = __ldg(u.c[0] + k);
  v[1] = __ldg(u.c[DIR == 0 ? 1 : 2] + k);
  v[2] = __ldg(u.c[DIR == 0 ? 2 : 1] + k);
  v[3] = __ldg(u.c[3] + k);
  v[4] = __ldg(u.c[4] + k);
  v[5] = __ldg((DIR == 0 ? u.byc : u.bxc) + k);
  v[6] = __ldg(u.c[7] + k);
}

// One warp's 32 faces (lane = face; `valid` false for lanes without one).
// All lanes of the warp must call it; `ws` is the warp's shared memory.
template <int DIR, int ORDER, bool EARLY = false>
__device__ void mp_faces_warp(const Grid& g, const StateP& u, const IfaceP& out, double gamma,
                              int i, int j, bool valid, double* ws) {
  constexpr int H = ORDER == 5 ? 2 : 3;
  constexpr int S = 2 * H + 2, W = 2 * H + 1;
  constexpr bool SHORT = ORDER == 7;
  const unsigned lane = threadIdx.x & 31u;
  const long long step = DIR == 0 ? 1 : g.pitch;
  const long long k0 = valid ? g.idx(i, j) : 0;
  double* rec = ws;
  const St cl = valid ? load_cell(u, k0 - step) : St{}, cr = valid ? load_cell(u, k0) : St{};
  // A warp whose faces all lie in uniform regions (ambient gas around a blast
  // or a rotor) is done without eigenvectors: every stencil delta is zero, so
  // both face states are the reference state bit for bit.  The density across
  // the face is tested first, where a developed flow stops after one
  // comparison and one vote.  Rotor 4096^2 MP7, per step: 22.4 -> 8.7 ms; flow
  // 2048^2: 5.68 -> 5.69.  (The rest reloads its cells: the common path keeps
  // no register for it.)  MP7 alone: the same test in the MP5 kernel, which
  // holds its stencil in flight, costs a flow 1% (1024^2: 1.383 -> 1.396).
  if (SHORT && __all_sync(0xffffffffu, cl.rho == cr.rho)) {
    bool flat = true;
    if (valid) {
#pragma unroll 1
      for (int t = -(H + 1); t <= H; ++t) {
        double a[7], b[7];
        cell7<DIR>(u, k0, a);
        cell7<DIR>(u, k0 + t * step, b);
#pragma unroll
        for (int v = 0; v < 7; ++v) flat = flat && a[v] == b[v];
      }
    }
    if (__all_sync(0xffffffffu, flat)) {
      if (valid) {
        const St a = load_cell(u, k0 - step);
        St c = load_cell(u, k0);
        c.bx = 0.5 * a.bx + 0.5 * c.bx;
        c.by = 0.5 * a.by + 0.5 * c.by;
        finish_face<DIR, ORDER, 0>(g, u, out, gamma, i, j, k0, step, c, c);
      }
      return;
    }
  }
  // phase 1: reference state and eigen scalars of this lane's face
  bool sure = true;
  if (valid) {
    St ref;
    ref.rho = 0.5 * cl.rho + 0.5 * cr.rho;
    ref.mx = 0.5 * cl.mx + 0.5 * cr.mx;
    ref.my = 0.5 * cl.my + 0.5 * cr.my;
    ref.mz = 0.5 * cl.mz + 0.5 * cr.mz;
    ref.E = 0.5 * cl.E + 0.5 * cr.E;
    ref.bx = 0.5 * cl.bx + 0.5 * cr.bx;
    ref.by = 0.5 * cl.by + 0.5 * cr.by;
    ref.bz = 0.5 * cl.bz + 0.5 * cr.bz;
    const St c = rot<DIR>(ref);
    const Eg e = eig_scalars(c, gamma);
    double* r = rec + lane;
    r[(kRecC + 0) * kRecS] = c.rho;
    r[(kRecC + 1) * kRecS] = c.mx;
    r[(kRecC + 2) * kRecS] = c.my;
    r[(kRecC + 3) * kRecS] = c.mz;
    r[(kRecC + 4) * kRecS] = c.E;
    r[(kRecC + 5) * kRecS] = c.bx;
    r[(kRecC + 6) * kRecS] = c.by;
    r[(kRecC + 7) * kRecS] = c.bz;
    const double ev[16] = {e.sr, e.cf, e.cs, e.a, e.af, e.as, e.b1, e.b2, e.sbn,
                           e.vn, e.vt1, e.vt2, e.ia2, e.ra2, e.hv2, e.ir};
    sure = e.sure;
#pragma unroll
    for (int q = 0; q < 16; ++q) r[(kRecE + q) * kRecS] = ev[q];
  }
  const unsigned vmask = __ballot_sync(0xffffffffu, valid);
  const unsigned smask = __ballot_sync(0xffffffffu, sure);
  __syncwarp();  // the records are written (a ballot orders no memory)
  // phase 2: eight faces per round, four lanes per face
  const int gi = int(lane >> 2), rl = int(lane & 3u);
  double* grp = ws + kRec * kRecS + gi * kGrpDoubles;
  const double gm1 = gamma - 1.0, igm = 1.0 / gm1;
  constexpr double kTol = 1024.0 * kEps;
#pragma unroll 1
  for (int rd = 0; rd < 4; ++rd) {
    if (((vmask >> (8 * rd)) & 0xFFu) == 0u) continue;  // warp-uniform
    const int f = 8 * rd + gi;
    const bool on = (vmask >> f) & 1u;
    const long long kf = __shfl_sync(0xffffffffu, k0, f);
    WavePair w;
    // the stencil cells rl and rl + 4 (canonical frame; the normal field is not
    // reconstructed).  EARLY: in flight while the wave vectors are formed
    // (MP5 1024^2: 1.46 -> 1.40 ms per step).  At MP7 and in the batched and
    // listed kernels that spills, and they are loaded where they are used
    // (MP7 2048^2: 5.7 against 6.3 ms; batched MP5 1.02 against 1.09).
    double ca[7], cb[7];
    auto load_cells = [&] {
      cell7<DIR>(u, kf + (long long)(rl - 1 - H) * step, ca);
      if (rl + 4 < S) cell7<DIR>(u, kf + (long long)(rl + 3 - H) * step, cb);
    };
    if (on) {
      if (EARLY) load_cells();
      const double* r = rec + f;
      Eg e;
      e.rho = r[(kRecC + 0) * kRecS];
      e.bt1 = r[(kRecC + 6) * kRecS];
      e.bt2 = r[(kRecC + 7) * kRecS];
      e.sr = r[(kRecE + 0) * kRecS];
      e.cf = r[(kRecE + 1) * kRecS];
      e.cs = r[(kRecE + 2) * kRecS];
      e.a = r[(kRecE + 3) * kRecS];
      e.af = r[(kRecE + 4) * kRecS];
      e.as = r[(kRecE + 5) * kRecS];
      e.b1 = r[(kRecE + 6) * kRecS];
      e.b2 = r[(kRecE + 7) * kRecS];
      e.sbn = r[(kRecE + 8) * kRecS];
      e.vn = r[(kRecE + 9) * kRecS];
      e.vt1 = r[(kRecE + 10) * kRecS];
      e.vt2 = r[(kRecE + 11) * kRecS];
      e.ia2 = r[(kRecE + 12) * kRecS];
      e.ra2 = r[(kRecE + 13) * kRecS];
      e.hv2 = r[(kRecE + 14) * kRecS];
      e.ir = r[(kRecE + 15) * kRecS];
      e.gm1 = gm1;
      e.igm = igm;
      wave_pair(e, rl, w);
      double2* col = reinterpret_cast<double2*>(grp + kPair * rl);
      col[0] = make_double2(w.rt[0], w.rt[1]);
      col[1] = make_double2(w.rt[2], w.rt[3]);
      col[2] = make_double2(w.rt[4], w.rt[5]);
      col[3] = make_double2(w.rt[6], 0.0);
      if (rl < 3) {
        col[4] = make_double2(w.rv[0], w.rv[1]);
        col[5] = make_double2(w.rv[2], w.rv[3]);
      }
    }
    __syncwarp();
    // L R = I within 1024 ulp (mhd_eigensystem.hpp:416-430), where no face of
    // the round is known to pass it: the four products of this lane's rows
    // T -+ V with a pair's columns are A + D -+ (B + C) and A - D +- (B - C), so
    // both members of each are within the tolerance where the sum of the two
    // magnitudes is
    bool usable = true;
    if (((smask >> (8 * rd)) & 0xFFu) != 0xFFu) {  // warp-uniform
      bool ok = true;
      if (on) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double2* R2 = reinterpret_cast<const double2*>(grp + kPair * q);
          const double2 p0 = R2[0], p1 = R2[1], p2 = R2[2], p3 = R2[3];
          const double A = fma(w.lt[0], p0.x, fma(w.lt[1], p0.y, fma(w.lt[2], p1.x, w.lt[3] * p1.y))) +
                           fma(w.lt[4], p2.x, fma(w.lt[5], p2.y, w.lt[6] * p3.x));
          const double C = fma(w.lv[0], p0.x, fma(w.lv[1], p0.y, fma(w.lv[2], p1.x, w.lv[3] * p1.y)));
          const double one = q == rl ? 1.0 : 0.0;
          if (q < 3) {
            const double2 v0 = R2[4], v1 = R2[5];
            const double B = fma(w.lt[1], v0.x, fma(w.lt[2], v0.y, fma(w.lt[3], v1.x, w.lt[4] * v1.y)));
            const double Dd = fma(w.lv[1], v0.x, fma(w.lv[2], v0.y, w.lv[3] * v1.x));
            ok = ok && fabs((A - one) + Dd) + fabs(B + C) <= kTol && fabs(A - Dd) + fabs(B - C) <= kTol;
          } else {
            ok = ok && fabs(A - one) + fabs(C) <= kTol;
          }
        }
      }
      const unsigned okm = __ballot_sync(0xffffffffu, ok);
      usable = ((okm >> (gi * 4)) & 0xFu) == 0xFu;
    }
    // stencil deltas of this lane's cells
    if (on) {
      if (!EARLY) load_cells();
      const double* r = rec + f;
      const double c7[7] = {r[(kRecC + 0) * kRecS], r[(kRecC + 1) * kRecS], r[(kRecC + 2) * kRecS],
                            r[(kRecC + 3) * kRecS], r[(kRecC + 4) * kRecS], r[(kRecC + 6) * kRecS],
                            r[(kRecC + 7) * kRecS]};
      double* dd = grp + kGrpD + rl * 7;
#pragma unroll
      for (int v = 0; v < 7; ++v) dd[v] = ca[v] - c7[v];
      if (rl + 4 < S) {
#pragma unroll
        for (int v = 0; v < 7; ++v) dd[28 + v] = cb[v] - c7[v];
      }
    }
    __syncwarp();
    // projection onto this lane's waves
    double cha[S], chb[S];
    if (on) {
#pragma unroll
      for (int sc = 0; sc < S; ++sc) {
        const double* dd = grp + kGrpD + sc * 7;
        if (usable) {
          const double d0 = dd[0], d1 = dd[1], d2 = dd[2], d3 = dd[3];
          const double t = fma(w.lt[0], d0, fma(w.lt[1], d1, fma(w.lt[2], d2, w.lt[3] * d3))) +
                           fma(w.lt[4], dd[4], fma(w.lt[5], dd[5], w.lt[6] * dd[6]));
          const double v = fma(w.lv[0], d0, fma(w.lv[1], d1, fma(w.lv[2], d2, w.lv[3] * d3)));
          cha[sc] = t - v;
          chb[sc] = t + v;
        } else {
          cha[sc] = dd[rl];
          chb[sc] = dd[6 - rl];
        }
      }
    }
    __syncwarp();  // the deltas are read; the face values overwrite them
    // MP limiter on both sides of both waves; kept as the sum and the
    // difference that multiply the pair's T and V columns
    if (on) {
      double al, ar, bl, br;
      mp_pair_limit<W>(cha, al, ar);
      if (rl < 3) mp_pair_limit<W>(chb, bl, br);
      else bl = br = 0.0;
      // (without usable eigenvectors wave r is component r and wave 6 - r
      // component 6 - r, kept unmixed)
      double2* x = reinterpret_cast<double2*>(grp + kGrpW + 2 * rl);
      x[0] = usable ? make_double2(al + bl, bl - al) : make_double2(al, bl);
      x[4] = usable ? make_double2(ar + br, br - ar) : make_double2(ar, br);
    }
    __syncwarp();
    // back-projection: lane rl forms components rl and rl + 4 of both sides
    if (on) {
      const double2* x2 = reinterpret_cast<const double2*>(grp + kGrpW);
      const double2 l0 = x2[0], l1 = x2[1], l2 = x2[2], l3 = x2[3];
      const double2 r0 = x2[4], r1 = x2[5], r2 = x2[6], r3 = x2[7];
      const int v1 = rl > 0 ? kPairV + rl - 1 : 7;  // V part of component rl (7: a zero)
      const double t0 = grp[rl], t1 = grp[kPair + rl], t2 = grp[2 * kPair + rl], t3 = grp[3 * kPair + rl];
      const double u0 = grp[v1], u1 = grp[kPair + v1], u2 = grp[2 * kPair + v1];
      double dl = fma(t0, l0.x, fma(t1, l1.x, fma(t2, l2.x, t3 * l3.x))) +
                  fma(u0, l0.y, fma(u1, l1.y, u2 * l2.y));
      double dr = fma(t0, r0.x, fma(t1, r1.x, fma(t2, r2.x, t3 * r3.x))) +
                  fma(u0, r0.y, fma(u1, r1.y, u2 * r2.y));
      if (!usable) {
        dl = rl == 0 ? l0.x : rl == 1 ? l1.x : rl == 2 ? l2.x : l3.x;
        dr = rl == 0 ? r0.x : rl == 1 ? r1.x : rl == 2 ? r2.x : r3.x;
      }
      rec[(kRecE + rl) * kRecS + f] = dl;
      rec[(kRecE + 7 + rl) * kRecS + f] = dr;
      if (rl < 3) {  // components 4, 5, 6; of these only the energy has a V part
        const double s0 = grp[rl + 4], s1 = grp[kPair + rl + 4], s2 = grp[2 * kPair + rl + 4],
                     s3 = grp[3 * kPair + rl + 4];
        double el = fma(s0, l0.x, fma(s1, l1.x, fma(s2, l2.x, s3 * l3.x)));
        double er = fma(s0, r0.x, fma(s1, r1.x, fma(s2, r2.x, s3 * r3.x)));
        if (rl == 0) {
          const double w0 = grp[kPairV + 3], w1 = grp[kPair + kPairV + 3],
                       w2 = grp[2 * kPair + kPairV + 3];
          el += fma(w0, l0.y, fma(w1, l1.y, w2 * l2.y));
          er += fma(w0, r0.y, fma(w1, r1.y, w2 * r2.y));
        }
        if (!usable) {
          el = rl == 0 ? l2.y : rl == 1 ? l1.y : l0.y;
          er = rl == 0 ? r2.y : rl == 1 ? r1.y : r0.y;
        }
        rec[(kRecE + 4 + rl) * kRecS + f] = el;
        rec[(kRecE + 11 + rl) * kRecS + f] = er;
      }
    }
    __syncwarp();
  }
  // phase 3: this lane's face
  if (!valid) return;
  const double* r = rec + lane;
  St c;
  c.rho = r[(kRecC + 0) * kRecS];
  c.mx = r[(kRecC + 1) * kRecS];
  c.my = r[(kRecC + 2) * kRecS];
  c.mz = r[(kRecC + 3) * kRecS];
  c.E = r[(kRecC + 4) * kRecS];
  c.bx = r[(kRecC + 5) * kRecS];
  c.by = r[(kRecC + 6) * kRecS];
  c.bz = r[(kRecC + 7) * kRecS];
  double dl[7], dr[7];
#pragma unroll
  for (int v = 0; v < 7; ++v) {
    dl[v] = r[(kRecE + v) * kRecS];
    dr[v] = r[(kRecE + 7 + v) * kRecS];
  }
  const St sl{c.rho + dl[0], c.mx + dl[1], c.my + dl[2], c.mz + dl[3],
              c.E + dl[4],   c.bx,         c.by + dl[5], c.bz + dl[6]};
  const St sr{c.rho + dr[0], c.mx + dr[1], c.my + dr[2], c.mz + dr[3],
              c.E + dr[4],   c.bx,         c.by + dr[5], c.bz + dr[6]};
  finish_face<DIR, ORDER, 0>(g, u, out, gamma, i, j, k0, step, rot<DIR>(sl), rot<DIR>(sr));
}

// ---- MUSCL-minmod in primitive variables (mhd_reconstruct.hip:93-404) ----
__device__ __forceinline__ int slope_drop(int c, int n, int lo, int hi) {
  if (lo != 0 && lo != 4 && c <= 0) return -1;
  if (hi != 0 && hi != 4 && c >= n - 1) return 1;
  return 0;
}
__device__ __forceinline__ double lim(double back, double fwd, int drop) {
  if (drop < 0) return fwd;
  if (drop > 0) return back;
  return minmod2(back, fwd);
}
__device__ __forceinline__ Pr muscl_face(const Pr& m, const Pr& c, const Pr& p, double sign,
                                         int drop) {
  const double h = 0.5 * sign;
  Pr f;
  f.rho = c.rho + h * lim(c.rho - m.rho, p.rho - c.rho, drop);
  f.vx = c.vx + h * lim(c.vx - m.vx, p.vx - c.vx, drop);
  f.vy = c.vy + h * lim(c.vy - m.vy, p.vy - c.vy, drop);
  f.vz = c.vz + h * lim(c.vz - m.vz, p.vz - c.vz, drop);
  f.p = c.p + h * lim(c.p - m.p, p.p - c.p, drop);
  f.bx = c.bx + h * lim(c.bx - m.bx, p.bx - c.bx, drop);
  f.by = c.by + h * lim(c.by - m.by, p.by - c.by, drop);
  f.bz = c.bz + h * lim(c.bz - m.bz, p.bz - c.bz, drop);
  return f;
}
template <int DIR>
__device__ void muscl_pair(const Grid& g, const StateP& u, int i, int j, long long k0,
                           long long step, double gamma, St& ul, St& ur) {
  const Pr a = to_prim(load_cell(u, k0 - 2 * step), gamma);
  const Pr b = to_prim(load_cell(u, k0 - step), gamma);
  const Pr c = to_prim(load_cell(u, k0), gamma);
  const Pr d = to_prim(load_cell(u, k0 + step), gamma);
  const int n = DIR == 0 ? g.nx : g.ny;
  const int lo = g.bc[DIR * 2], hi = g.bc[DIR * 2 + 1];
  const int pos = DIR == 0 ? i : j;
  const double igm = 1.0 / (gamma - 1.0);
  ul = to_cons(muscl_face(a, b, c, 1.0, slope_drop(pos - 1, n, lo, hi)), igm);
  ur = to_cons(muscl_face(b, c, d, -1.0, slope_drop(pos, n, lo, hi)), igm);
}

// How far the limited characteristic face state departs from the unlimited
// component-wise one: the largest difference relative to the state's scale
// per group (rho; momentum against sqrt(2 rho E); E; field against
// sqrt(2 E)); +inf when not finite.
__device__ __forceinline__ float limiter_departure(const St& a, const St& b) {
  const double rs = fabs(b.rho), es = fabs(b.E);
  const double ms = sqrt(2.0 * rs * es), bs = sqrt(2.0 * es);
  double d = fabs(a.rho - b.rho) / rs;
  d = fmax(d, fabs(a.mx - b.mx) / ms);
  d = fmax(d, fabs(a.my - b.my) / ms);
  d = fmax(d, fabs(a.mz - b.mz) / ms);
  d = fmax(d, fabs(a.E - b.E) / es);
  d = fmax(d, fabs(a.bx - b.bx) / bs);
  d = fmax(d, fabs(a.by - b.by) / bs);
  d = fmax(d, fabs(a.bz - b.bz) / bs);
  return isfinite(d) ? float(d) : INFINITY;
}

// Learned-mode face list of one direction: the per-cell flags it was built
// from (a face is listed when either of its cells is flagged), the list and
// its device-resident count.
struct FaceList {
  const unsigned char* flag;
  int* list;
  int* count;
};

// One face's interface states.  MODE 0: the characteristic MP path; 1: the
// same, also recording per cell the largest departure of a limited state
// from the unlimited component-wise one (label[cell] = max, as float bits;
// the left state's stencil is centred on the left cell);
// 2: the unlimited component-wise path; a face whose unlimited states are
// not admissible is appended to `defer` for the characteristic pass that
// follows (the plain step's path for it, fallbacks included) unless it is
// listed already; 3: the characteristic path, recording per cell whether the
// MP limiter fired on any characteristic field of a state whose stencil is
// centred on it (label[cell] = 1).  Orders 1 and 2 ignore MODE.
template <int DIR, int ORDER, int MODE>
__device__ __forceinline__ void recon_face(const Grid& g, const StateP& u, const IfaceP& out,
                                           double gamma, int i, int j, int* label,
                                           FaceList defer = FaceList{}) {
  const long long k0 = g.idx(i, j);
  const long long step = DIR == 0 ? 1 : g.pitch;
  St ul, ur;
  if (ORDER <= 1) {
    ul = DIR == 0 ? load_cell1(u, g, i - 1, j) : load_cell1(u, g, i, j - 1);
    ur = load_cell1(u, g, i, j);
  } else if (ORDER == 2) {
    muscl_pair<DIR>(g, u, i, j, k0, step, gamma, ul, ur);
  } else {
    constexpr int H = ORDER == 5 ? 2 : 3;
    if constexpr (MODE == 2) {
      mp_pair_lin<DIR, H>(u, k0, step, ul, ur);
      if (!recon_admissible(ul, gamma) || !recon_admissible(ur, gamma)) {
        if (!defer.flag[k0 - step] && !defer.flag[k0])
          defer.list[atomicAdd(defer.count, 1)] = int(k0);
        return;
      }
    } else {
      bool fl = false, fr = false;
      mp_pair_loop<DIR, H>(u, k0, step, gamma, ul, ur, &fl, &fr);
      if (MODE == 3) {
        // the literal label: the MP limiter fired on some characteristic
        // field of the state whose stencil is centred on the cell
        if (fl) atomicMax(label + (k0 - step), 1);
        if (fr) atomicMax(label + k0, 1);
      }
      if (MODE == 1) {
        St ll, lr;
        mp_pair_lin<DIR, H>(u, k0, step, ll, lr);
        // non-negative floats order like their bit patterns
        atomicMax(label + (k0 - step), __float_as_int(limiter_departure(ul, ll)));
        atomicMax(label + k0, __float_as_int(limiter_departure(ur, lr)));
      }
    }
  }
  finish_face<DIR, ORDER, MODE>(g, u, out, gamma, i, j, k0, step, ul, ur);
}

// The fallback chain after the high-order states of one face
// (mhd_reconstruct.hip:514-670): MUSCL when a characteristic MP state is not
// admissible, the shared CT normal field, first order, then NaN; the states
// are written to the face's interface slots.
template <int DIR, int ORDER, int MODE>
__device__ __forceinline__ void finish_face(const Grid& g, const StateP& u, const IfaceP& out,
                                            double gamma, int i, int j, long long k0,
                                            long long step, St ul, St ur) {
  if constexpr (ORDER >= 5 && MODE != 2) {
    if (!recon_admissible(ul, gamma) || !recon_admissible(ur, gamma))
      muscl_pair<DIR>(g, u, i, j, k0, step, gamma, ul, ur);
  }
  const double bn = (DIR == 0 ? u.c[5] : u.c[6])[k0];
  set_normal_b<DIR>(ul, bn);
  set_normal_b<DIR>(ur, bn);
  if (!recon_admissible(ul, gamma) || !recon_admissible(ur, gamma)) {
    if (ORDER <= 1) {
      ul = DIR == 0 ? load_cell1(u, g, i - 1, j) : load_cell1(u, g, i, j - 1);
      ur = load_cell1(u, g, i, j);
    } else {
      ul = load_cell(u, k0 - step);
      ur = load_cell(u, k0);
    }
    set_normal_b<DIR>(ul, bn);
    set_normal_b<DIR>(ur, bn);
  }
  if (!(recon_admissible(ul, gamma) || subnormal_admissible(ul)) ||
      !(recon_admissible(ur, gamma) || subnormal_admissible(ur))) {
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    ul = St{nan, nan, nan, nan, nan, nan, nan, nan};
    ur = ul;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    out.L[c][k0] = comp(ul, c);
    out.R[c][k0] = comp(ur, c);
  }
}

template <int DIR, int ORDER, int MODE = 0, bool EARLY = false>
__device__ __forceinline__ void b_reconstruct(const Grid& g, const StateP& u, const IfaceP& out,
                                              double gamma, const Ctl* ctl, int bx, int by,
                                              int* label = nullptr,
                                              FaceList defer = FaceList{}) {
  // dir 0: faces i in [0,nx] over all padded rows; dir 1: transposed.
  const int i = bx * blockDim.x + threadIdx.x - (DIR == 1 ? g.ng : 0);
  const int j = by * blockDim.y + threadIdx.y - (DIR == 0 ? g.ng : 0);
  const bool valid = !(DIR == 0 ? (i > g.nx || j >= g.ny + g.ng) : (i >= g.nx + g.ng || j > g.ny));
  if (ctl->status & ~kStatusDone) return;  // uniform: no kernel of a step writes it mid-launch
  if constexpr (MODE == 0 && ORDER >= 5) {
    // the characteristic path, warp-cooperative (threadIdx.y = warp)
    extern __shared__ double dsm[];
    mp_faces_warp<DIR, ORDER, EARLY>(g, u, out, gamma, i, j, valid,
                                     dsm + threadIdx.y * kWarpReconDoubles);
    return;
  }
  if (!valid) return;
  recon_face<DIR, ORDER, MODE>(g, u, out, gamma, i, j, label, defer);
}

// The faces of one direction (dir0 + blockIdx.z) or, with two layers of
// blocks, of both in one launch: the y faces' blocks fill the SMs while the x
// faces' last ones drain, and a grid that does not fill the chip (a 64^2 grid
// has 37 blocks a direction) runs both side by side.  64^2 MP5 step 0.26 ->
// 0.21 ms with the face flux launched the same way.
template <int ORDER>
__global__ void __launch_bounds__(128, 4) k_reconstruct(Grid g, StateP u, IfaceP ix, IfaceP iy,
                                                        double gamma, const Ctl* ctl, int dir0) {
  if (dir0 + int(blockIdx.z) == 0)
    b_reconstruct<0, ORDER, 0, ORDER == 5>(g, u, ix, gamma, ctl, blockIdx.x, blockIdx.y);
  else
    b_reconstruct<1, ORDER, 0, ORDER == 5>(g, u, iy, gamma, ctl, blockIdx.x, blockIdx.y);
}

// Limiter labels of the cells (training data of the indicator): the
// departure of the limited states (literal = 0) or whether the limiter fired
// (literal = 1).
template <int DIR, int ORDER>
__global__ void __launch_bounds__(128) k_reconstruct_label(Grid g, StateP u, IfaceP out,
                                                           double gamma, const Ctl* ctl,
                                                           int* label, int literal) {
  if (literal)
    b_reconstruct<DIR, ORDER, 3>(g, u, out, gamma, ctl, blockIdx.x, blockIdx.y, label);
  else
    b_reconstruct<DIR, ORDER, 1>(g, u, out, gamma, ctl, blockIdx.x, blockIdx.y, label);
}

// Learned mode, pass 1: every face by the unlimited component-wise path
// (inadmissible ones deferred to pass 2).  Memory-latency bound: at 64
// registers and eight blocks per SM it ran 17% faster than at 94 and five.
// mp_pair_lin from a shared-memory tile: component v's stencil cell t at
// tile[v pc + pos + t tstep]; the same operations in the same order.
template <int DIR, int H>
__device__ __forceinline__ void mp_pair_lin_tile(const double* tile, int pc, int pos, int tstep,
                                                 St& ul, St& ur) {
  constexpr int S = 2 * H + 2, W = 2 * H + 1;
  double dl[8], dr[8], cv[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const double* a = tile + v * pc + pos;
    const double c = 0.5 * a[H * tstep] + 0.5 * a[(H + 1) * tstep];
    cv[v] = c;
    if (v == 5) continue;  // the normal field is not reconstructed
    double w[S];
#pragma unroll
    for (int t = 0; t < S; ++t) w[t] = a[t * tstep] - c;
    dl[v] = mp_interp_plain<W>(w);
    double wr[W];
#pragma unroll
    for (int t = 0; t < W; ++t) wr[t] = w[W - t];
    dr[v] = mp_interp_plain<W>(wr);
  }
  const St sl{cv[0] + dl[0], cv[1] + dl[1], cv[2] + dl[2], cv[3] + dl[3],
              cv[4] + dl[4], cv[5],         cv[6] + dl[6], cv[7] + dl[7]};
  const St sr{cv[0] + dr[0], cv[1] + dr[1], cv[2] + dr[2], cv[3] + dr[3],
              cv[4] + dr[4], cv[5],         cv[6] + dr[6], cv[7] + dr[7]};
  ul = rot<DIR>(sl);
  ur = rot<DIR>(sr);
}

// The block's stencil cells (canonical components) are staged in shared
// memory once, each read by up to 2H + 2 faces (5.7 -> 5.0 ms of component-wise
// and listed passes per learned rotor 4096^2 MP7 step, the state
// bit-identical).  Every stencil cell of a valid face lies inside the padded
// grid, so the staged values are the ones the per-face loads read.
template <int DIR, int ORDER>
__global__ void __launch_bounds__(128, 8) k_reconstruct_lin(Grid g, StateP u, IfaceP out,
                                                         double gamma, const Ctl* ctl,
                                                         FaceList defer) {
  constexpr int H = ORDER == 5 ? 2 : 3, S = 2 * H + 2;
  constexpr int TW = DIR == 0 ? kBX + S - 1 : kBX;  // staged columns
  constexpr int TH = DIR == 0 ? 4 : 4 + S - 1;      // staged rows
  constexpr int PC = TW * TH;
  __shared__ double tile[8 * PC];
  if (ctl->status & ~kStatusDone) return;  // uniform: no kernel of a step writes it mid-launch
  const int i0 = blockIdx.x * kBX - (DIR == 1 ? g.ng : 0);
  const int j0 = blockIdx.y * 4 - (DIR == 0 ? g.ng : 0);
  const int ci0 = DIR == 0 ? i0 - 1 - H : i0, cj0 = DIR == 0 ? j0 : j0 - 1 - H;
  const int tid = threadIdx.y * kBX + threadIdx.x;
  for (int e = tid; e < PC; e += kBX * 4) {
    const int r = e / TW, c = e - r * TW;
    const int ci = ci0 + c, cj = cj0 + r;
    const bool in = ci >= -g.ng && ci < g.nx + g.ng && cj >= -g.ng && cj < g.ny + g.ng;
    const long long k = in ? g.idx(ci, cj) : 0;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const double* a = v == 0 ? u.c[0]
                        : v == 1 ? (DIR == 0 ? u.c[1] : u.c[2])
                        : v == 2 ? (DIR == 0 ? u.c[2] : u.c[1])
                        : v == 3 ? u.c[3]
                        : v == 4 ? u.c[4]
                        : v == 5 ? (DIR == 0 ? u.bxc : u.byc)
                        : v == 6 ? (DIR == 0 ? u.byc : u.bxc)
                                 : u.c[7];
      tile[v * PC + e] = in ? __ldg(a + k) : 0.0;
    }
  }
  __syncthreads();
  const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
  const bool valid = !(DIR == 0 ? (i > g.nx || j >= g.ny + g.ng) : (i >= g.nx + g.ng || j > g.ny));
  if (!valid) return;
  const long long k0 = g.idx(i, j);
  const long long step = DIR == 0 ? 1 : g.pitch;
  St ul, ur;
  mp_pair_lin_tile<DIR, H>(tile, PC, threadIdx.y * TW + threadIdx.x, DIR == 0 ? 1 : TW, ul, ur);
  if (!recon_admissible(ul, gamma) || !recon_admissible(ur, gamma)) {
    if (!defer.flag[k0 - step] && !defer.flag[k0]) defer.list[atomicAdd(defer.count, 1)] = int(k0);
    return;
  }
  finish_face<DIR, ORDER, 2>(g, u, out, gamma, i, j, k0, step, ul, ur);
}

// Learned mode, pass 2: the listed faces (padded linear index of the face's
// high cell) by the full characteristic path; the count is read on the device.
// Warps take 32 consecutive list entries at a time.
template <int DIR, int ORDER>
__device__ __forceinline__ void b_reconstruct_list(const Grid& g, const StateP& u,
                                                   const IfaceP& out, double gamma,
                                                   const int* list, int n) {
  extern __shared__ double dsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* ws = dsm + warp * kWarpReconDoubles;
  for (int base = (blockIdx.x * kReconWarps + warp) * 32; base < n;
       base += gridDim.x * kReconWarps * 32) {
    const int t = base + lane;
    const bool valid = t < n;
    int i = 0, j = 0;
    if (valid) {
      const int k = list[t];
      i = k % g.pitch - g.ng;
      j = k / g.pitch - g.ng;
    }
    mp_faces_warp<DIR, ORDER>(g, u, out, gamma, i, j, valid, ws);
  }
}

template <int DIR, int ORDER>
__global__ void __launch_bounds__(128, 4) k_reconstruct_list(Grid g, StateP u, IfaceP out,
                                                             double gamma, const Ctl* ctl,
                                                             const int* list, const int* count) {
  if (ctl->status & ~kStatusDone) return;
  b_reconstruct_list<DIR, ORDER>(g, u, out, gamma, list, *count);
}

// Faces whose either cell is flagged, appended to the x and y lists in
// warp-aggregated order; padded cells are scanned row-major.
__global__ void k_face_lists(Grid g, const unsigned char* flag, int* xlist, int* ylist,
                             int* counts) {
  const long long n = g.size();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const unsigned lane = threadIdx.x & 31;
  bool nx_ = false, ny_ = false;
  int k = 0;
  if (t < n) {
    k = int(t);
    const int i = int(t % g.pitch) - g.ng, j = int(t / g.pitch) - g.ng;
    if (i >= 0 && i <= g.nx && j < g.ny + g.ng) nx_ = (flag[t] | flag[t - 1]) != 0;
    if (j >= 0 && j <= g.ny && i < g.nx + g.ng) ny_ = (flag[t] | flag[t - g.pitch]) != 0;
  }
  const unsigned bx_ = __ballot_sync(0xffffffffu, nx_), by_ = __ballot_sync(0xffffffffu, ny_);
  int basex = 0, basey = 0;
  if (lane == 0) {
    if (bx_) basex = atomicAdd(&counts[0], __popc(bx_));
    if (by_) basey = atomicAdd(&counts[1], __popc(by_));
  }
  basex = __shfl_sync(0xffffffffu, basex, 0);
  basey = __shfl_sync(0xffffffffu, basey, 0);
  const unsigned below = (1u << lane) - 1u;
  if (nx_) xlist[basex + __popc(bx_ & below)] = k;
  if (ny_) ylist[basey + __popc(by_ & below)] = k;
}


}  // namespace

// ===========================================================================
// Face flux (mhd_riemann.hip:53-136, mhd_face_quadrature.hpp:114-273) with
// the CT face EMF of the same solve (mhd_ct.hip:330-359) and the CFL face
// signal speed (mhd_reduce.hip:254-416).
// ===========================================================================
namespace {

struct Spd {
  double v, f2;
};

// One side's |v_n| and squared fast speed (mhd_reduce.hip:254-325), with the
// reciprocal of rho.  The discriminant is formed as (a^2 - b^2)^2 + 4 a^2 b_t^2,
// which equals the reference's (a^2 + b^2)^2 - 4 a^2 b_n^2 but has no
// cancellation: where the reference's rounding is amplified to sqrt(eps) (a
// degenerate fan, a == b_n with b_t == 0) this form stays accurate to a few
// ulps, and elsewhere both agree to rounding.  A non-finite component makes
// the pressure fail its test (point_admissible_p).
template <int DIR>
__device__ __forceinline__ Spd speed_parts(const St& s, double gamma, double ir) {
  const double p = pressure_f(s, gamma, ir);
  if (!point_admissible_p(s, p)) return Spd{kInf, kInf};
  const double bn = DIR == 0 ? s.bx : s.by, b1 = DIR == 0 ? s.by : s.bx;
  const double a2 = gamma * p * ir;
  const double bn2 = bn * bn * ir;
  const double bt2 = (b1 * b1 + s.bz * s.bz) * ir;
  const double d = a2 - (bn2 + bt2);
  const double disc = d * d + 4.0 * a2 * bt2;
  return Spd{fabs(DIR == 0 ? s.mx : s.my) * ir, 0.5 * ((a2 + bn2 + bt2) + sqrt_nr(disc))};
}

// Weighted face rate 0.5*alpha/h of one Riemann problem (mhd_reduce.hip:331-383).
template <int DIR, int ORDER>
__device__ __forceinline__ double face_rate(const St& l, const St& r, double gamma, double h,
                                            double irl, double irr) {
  const Spd a = speed_parts<DIR>(l, gamma, irl), b = speed_parts<DIR>(r, gamma, irr);
  // a side whose discriminant overflows has NaN here, which a maximum would drop
  if (!(a.f2 < kInf && b.f2 < kInf)) return kInf;
  const double rate = ORDER <= 1 ? fmax(a.v + sqrt_nr(a.f2), b.v + sqrt_nr(b.f2))
                                 : fmax(a.v, b.v) + sqrt_nr(fmax(a.f2, b.f2));
  if (!(isfinite(rate) && rate >= 0.0)) return kInf;
  return div_by(rate * 0.5, h, pow2_recip(h));
}

__device__ __forceinline__ St iface(const IfaceP& v, long long k, bool left) {
  if (left)
    return St{__ldg(v.L[0] + k), __ldg(v.L[1] + k), __ldg(v.L[2] + k), __ldg(v.L[3] + k),
              __ldg(v.L[4] + k), __ldg(v.L[5] + k), __ldg(v.L[6] + k), __ldg(v.L[7] + k)};
  return St{__ldg(v.R[0] + k), __ldg(v.R[1] + k), __ldg(v.R[2] + k), __ldg(v.R[3] + k),
            __ldg(v.R[4] + k), __ldg(v.R[5] + k), __ldg(v.R[6] + k), __ldg(v.R[7] + k)};
}

// Orders 1 and 2, whose face states need no transverse quadrature: one thread
// per face.
template <int DIR, int ORDER>
__global__ void __launch_bounds__(128) k_face_flux(Grid g, IfaceP in, FluxP out, double* emf,
                                                   int* nj, double* spd, double gamma,
                                                   const Ctl* ctl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i > g.nx || j > g.ny) return;
  if (ctl->status & ~kStatusDone) return;
  int si = i, sj = j;
  // The periodic high face repeats face 0's Riemann data bit for bit.
  if (DIR == 0 && i == g.nx && g.bc[0] == 0 && g.bc[1] == 0) si = 0;
  if (DIR == 1 && j == g.ny && g.bc[2] == 0 && g.bc[3] == 0) sj = 0;
  const long long k = g.idx(i, j), ks = g.idx(si, sj);
  const St bl = iface(in, ks, true), br = iface(in, ks, false);
  const Fx f = riemann<DIR>(bl, br, ORDER <= 1, gamma);
  // out, emf and nj may each be absent (the per-kernel launch interface
  // asks for fluxes or for the CT face tables alone)
  if (out.f[0]) {
    out.f[0][k] = f.rho;
    out.f[1][k] = f.mx;
    out.f[2][k] = f.my;
    out.f[3][k] = f.mz;
    out.f[4][k] = f.E;
    out.f[5][k] = f.bx;
    out.f[6][k] = f.by;
    out.f[7][k] = f.bz;
  }
  // Directional Godunov E_z: F_x(By) = -Ez, F_y(Bx) = +Ez (mhd_ct.hip:126-133).
  if (emf) emf[k] = DIR == 0 ? -f.by : f.bx;
  if (spd)
    spd[k] = face_rate<DIR, ORDER>(bl, br, gamma, DIR == 0 ? g.dx : g.dy, rcp_rho(bl.rho),
                                   rcp_rho(br.rho));
  if (!nj) return;
  // "No jump" proof of the face's problem (mhd_ct.hip:150-174), mapped like
  // every CT table read.
  const long long km = g.idx(face_index(i, g.nx, g.bc[0], g.bc[1]),
                             face_index(j, g.ny, g.bc[2], g.bc[3]));
  int proof = 1;
#pragma unroll
  for (int c = 0; c < 8; ++c)
    if (!(in.L[c][km] == in.R[c][km])) proof = 0;
  nj[k] = proof;
}

}  // namespace

// ---------------------------------------------------------------------------
// MP5/MP7 face flux with one lane per Gauss point: a group of Q lanes owns a
// face (Q = 3 at MP5, 4 at MP7).  The interface states of a face tile (8 x 4
// at MP7, 8 x 5 at MP5) and its transverse halo are staged in shared memory,
// so each stencil row is read from L2 once per tile instead of once per face
// row (2.8x fewer for x faces, 4x for y faces at MP7).  At MP7 the
// transverse recovery is split by component: lane q forms components q,
// q + 4, ... at every Gauss point of its face (each stencil column read
// once) into the face's point rows in shared memory, from which each lane
// takes its own point's 16 components as 16-byte pairs.  Each lane solves its point's Riemann problem, the group
// votes on admissibility, and the point fluxes go back through the same
// rows, where lane q forms and stores the Gauss sums of components q, q + 4
// (rotor 4096^2 MP7: face flux 27.6 -> 23.3 ms per step; Orszag-Tang 2048^2
// MP7: 10.8 -> 10.4).  At MP5 each lane recovers its own point (below).
// 128 threads
// (smaller blocks than 16 x 4 measured 3-5% faster at MP7: a block waiting
// at the staging barrier holds fewer warps).
// ---------------------------------------------------------------------------
namespace {

constexpr int kFqTX = 8, kFqTY = 4;
// One lane per Gauss point: groups of 4 lanes (MP7, 8 faces per warp, 8 x 4
// face tiles) or 3 lanes (MP5, 10 faces per warp with two lanes idle, 8 x 5
// tiles); four warps per block either way.
constexpr int kFqThreads = 4 * kFqTX * kFqTY;
template <int ORDER>
constexpr int fq_ty() { return ORDER == 5 ? 5 : 4; }
// 96 registers (ptxas keeps a few values of the HLLD tail on the stack):
// five 128-thread blocks per SM measured 8-11% faster than four at 128
// registers (six spill more and lose it again).
constexpr int kFqBlocksPerSm = 5;
// Shared-memory strides in doubles.  A component plane of the tile is padded
// to 4 mod 16 doubles, so that the lanes of a group (components 4 apart of
// one cell) and the neighbouring groups (neighbouring cells) read distinct
// banks; a point row is 16 components + 2 (16-byte aligned), a face's rows
// are Q rows + 4.
constexpr int fq_plane(int cells) { return cells + ((4 - cells % 16) + 16) % 16; }
constexpr int kFqRow = 18;
template <int ORDER>
constexpr int fq_face() { return (ORDER == 5 ? 3 : 4) * kFqRow + 4; }

// All 2H + 1 transverse taps of a face staged with L == R in every component,
// from the tile's bits: the taps are N consecutive slots from s0 (y faces) or
// every TC-th one (x faces).
template <int DIR, int N>
__device__ __forceinline__ bool stencil_flat(const unsigned* same, int s0, int TC) {
  if (DIR == 1) {
    const unsigned b = __funnelshift_r(same[s0 >> 5], same[(s0 >> 5) + 1], s0 & 31);
    return (b & ((1u << N) - 1u)) == (1u << N) - 1u;
  }
  unsigned all = 1u;
#pragma unroll
  for (int t = 0; t < N; ++t) all &= same[(s0 + t * TC) >> 5] >> ((s0 + t * TC) & 31);
  return all & 1u;
}
// Flux of a point whose two sides are the same state: the physical flux.
template <int DIR>
__device__ __forceinline__ Fx flat_flux(const St& s, double p, double ir) {
  Fx f = physical_flux_xp(rot<DIR>(s), p, ir);
  if (DIR == 1) {
    const double t = f.mx;
    f.mx = f.my;
    f.my = t;
    f.bx = f.by;
    f.by = 0.0;
  }
  return f;
}

// All of a tile's n slot bits set.
template <int n>
__device__ __forceinline__ bool stencil_words(const unsigned* same) {
  bool all = true;
#pragma unroll
  for (int w = 0; w < (n + 31) / 32; ++w) {
    const unsigned full = n - 32 * w >= 32 ? ~0u : (1u << (n - 32 * w)) - 1u;
    all = all && same[w] == full;
  }
  return all;
}
// A tile whose staged states are all one state (uniform gas): every Gauss
// point of every face is that state, so the flux is its physical flux, the
// rate its own and the no-jump proof holds; one thread per face.  Only for
// tiles without mapped taps.  Rotor 4096^2 MP7: face flux 18.8 -> 13.4 ms per
// step, flow 2048^2 unchanged (5.24).  `at`: shared offset of component c of slot 0.
template <int DIR, int ORDER, int TX, class At>
__device__ __forceinline__ void constant_tile_flux(const Grid& g, const FluxP& out, double* emf,
                                                   int* nj, double* spd, double gamma, int i0,
                                                   int j0, At at) {
  constexpr int TY = fq_ty<ORDER>();
  const int f = threadIdx.x, i = i0 + f % TX, j = j0 + f / TX;
  if (f >= TX * TY || i > g.nx || j > g.ny) return;
  const long long k = g.idx(i, j);
  const St u{at(0), at(1), at(2), at(3), at(4), at(5), at(6), at(7)};
  const double ir = rcp_rho(u.rho);
  const Fx v = flat_flux<DIR>(u, pressure_f(u, gamma, ir), ir);
  if (out.f[0]) {
    out.f[0][k] = v.rho;
    out.f[1][k] = v.mx;
    out.f[2][k] = v.my;
    out.f[3][k] = v.mz;
    out.f[4][k] = v.E;
    out.f[5][k] = v.bx;
    out.f[6][k] = v.by;
    out.f[7][k] = v.bz;
  }
  if (emf) emf[k] = DIR == 0 ? -v.by : v.bx;
  if (spd) spd[k] = face_rate<DIR, ORDER>(u, u, gamma, DIR == 0 ? g.dx : g.dy, ir, ir);
  if (nj) nj[k] = 1;
}

// Per-point recovery (MP5): each lane forms all 16 components of its own
// Gauss point from the staged tile, and the group gathers the point fluxes
// by shuffles.  With three lanes per face the component split below leaves
// a lane with six components against five and measured 8% slower on
// Orszag-Tang 2048^2 MP5 (face flux 9.1 -> 9.8 ms per step).
template <int DIR, int ORDER, int TX = kFqTX>
__device__ __forceinline__ void b_face_flux_pt(const Grid& g, const IfaceP& in, const FluxP& out,
                                               double* emf, int* nj, double* spd, double gamma,
                                               const Ctl* ctl, int bx, int by, double* sm) {
  constexpr int H = ORDER == 5 ? 2 : 3, N = 2 * H + 1, Q = ORDER == 5 ? 3 : 4;
  constexpr int FPW = 32 / Q, TY = fq_ty<ORDER>();         // faces per warp, tile rows
  static_assert(4 * FPW == TX * TY, "four warps cover the face tile");
  constexpr int TR = DIR == 0 ? TY + 2 * H : TY;          // tile rows (j)
  constexpr int TC = DIR == 0 ? TX : TX + 2 * H;          // tile columns (i)
  double(*tile)[TR][TC] = reinterpret_cast<double(*)[TR][TC]>(sm);
  // staged and L == R in every component: one bit per tile slot
  constexpr int kWords = (TR * TC + 31) / 32;
  unsigned* same = reinterpret_cast<unsigned*>(sm + 16 * TR * TC);
  if (ctl->status) return;  // uniform over the block
  const int i0 = bx * TX, j0 = by * TY;
  const bool perx = g.bc[0] == 0 && g.bc[1] == 0, pery = g.bc[2] == 0 && g.bc[3] == 0;
  static_assert(TR * TC <= kFqThreads, "one tile slot per thread");
  {
    const int e = threadIdx.x;
    const int row = e / TC, col = e - row * TC;
    int fi, fj;
    bool valid;
    if (DIR == 0) {
      const int ii = i0 + col;
      fi = (ii == g.nx && perx) ? 0 : ii;
      fj = j0 - H + row;
      valid = e < TR * TC && ii <= g.nx && fj >= -g.ng && fj < g.ny + g.ng;
    } else {
      const int jj = j0 + row;
      fj = (jj == g.ny && pery) ? 0 : jj;
      fi = i0 - H + col;
      valid = e < TR * TC && jj <= g.ny && fi >= -g.ng && fi < g.nx + g.ng;
    }
    const long long kk = valid ? g.idx(fi, fj) : 0;
    bool eq = valid;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double a = valid ? __ldg(in.L[c] + kk) : 0.0;
      const double b = valid ? __ldg(in.R[c] + kk) : 0.0;
      if (e < TR * TC) {
        tile[c][row][col] = a;
        tile[8 + c][row][col] = b;
      }
      eq = eq && a == b;
    }
    const unsigned w = __ballot_sync(0xffffffffu, eq);
    if ((e & 31) == 0 && e / 32 < kWords) same[e / 32] = w;
    if (e == 0) same[kWords] = 0u;
  }
  __syncthreads();
  constexpr bool kLF = false;
  const int wl = threadIdx.x & 31;
  if (wl >= FPW * Q) return;  // the lanes no group uses (MP5)
  const int lane = wl % Q, base = wl - lane;
  const unsigned gmask = ((1u << Q) - 1u) << base;
  const int face = (threadIdx.x >> 5) * FPW + wl / Q;
  const int fx = face % TX, fy = face / TX;
  const int i = i0 + fx, j = j0 + fy;
  if (i > g.nx || j > g.ny) return;  // whole groups leave together
  const long long k = g.idx(i, j);
  const double h = DIR == 0 ? g.dx : g.dy;
  // tile coordinates of stencil tap t (t = H is the face itself)
  auto tr = [&](int t) { return DIR == 0 ? fy + t : fy; };
  auto tcl = [&](int t) { return DIR == 0 ? fx : fx + t; };
  auto slot = [&](int t) { return tr(t) * TC + tcl(t); };
  const bool flat = stencil_flat<DIR, N>(same, slot(0), TC);
  St l{}, r{};
  double irl = 1.0, irr = 1.0, prl = 0.0, prr = 0.0;
  bool ok = true;
  {
    double w[N];
#pragma unroll
    for (int t = 0; t < N; ++t) w[t] = point_w<ORDER>(lane, t);
    double pl[8], pr[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      double sa[N], sb[N];
#pragma unroll
      for (int t = 0; t < N; ++t) {
        sa[t] = tile[c][tr(t)][tcl(t)];
        sb[t] = tile[8 + c][tr(t)][tcl(t)];
      }
      pl[c] = wsum<N>(w, sa);
      pr[c] = wsum<N>(w, sb);
    }
    l = St{pl[0], pl[1], pl[2], pl[3], pl[4], pl[5], pl[6], pl[7]};
    r = St{pr[0], pr[1], pr[2], pr[3], pr[4], pr[5], pr[6], pr[7]};
    irl = rcp_nr(l.rho);
    irr = rcp_nr(r.rho);
    prl = pressure_f(l, gamma, irl);
    prr = pressure_f(r, gamma, irr);
    ok = point_admissible_p(l, prl) && point_admissible_p(r, prr);
  }
  auto centre = [&](bool left) {
    const int o = left ? 0 : 8, rr = tr(H), cc = tcl(H);
    return St{tile[o][rr][cc],     tile[o + 1][rr][cc], tile[o + 2][rr][cc], tile[o + 3][rr][cc],
              tile[o + 4][rr][cc], tile[o + 5][rr][cc], tile[o + 6][rr][cc], tile[o + 7][rr][cc]};
  };
  const unsigned bad = (__ballot_sync(gmask, !ok) >> base) & ((1u << Q) - 1u);
  const bool group_ok = bad == 0;
  const int first_bad = bad ? __ffs(bad) - 1 : Q;
  double rate = 0.0;
  if (spd) {
    if (lane == 0) {
      const St a = centre(true), b = centre(false);
      rate = face_rate<DIR, ORDER>(a, b, gamma, h, rcp_rho(a.rho), rcp_rho(b.rho));
    }
    if (lane < first_bad) rate = fmax(rate, face_rate<DIR, ORDER>(l, r, gamma, h, irl, irr));
  }
  const bool solve = group_ok || lane == 0;
  if (!group_ok) {
    l = centre(true);
    r = centre(false);
    irl = rcp_rho(l.rho);
    irr = rcp_rho(r.rho);
    prl = pressure_f(l, gamma, irl);
    prr = pressure_f(r, gamma, irr);
  }
  double fv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (solve) {
    const Fx f = flat ? flat_flux<DIR>(l, prl, irl) : riemann<DIR, false>(l, r, kLF, gamma, irl, irr, prl, prr);
    fv[0] = f.rho; fv[1] = f.mx; fv[2] = f.my; fv[3] = f.mz;
    fv[4] = f.E;   fv[5] = f.bx; fv[6] = f.by; fv[7] = f.bz;
  }
  double res[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if (group_ok) {
      double sq[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) sq[q] = __shfl_sync(gmask, fv[c], base + q);
      res[c] = gauss_avg<ORDER>(sq);
    } else {
      res[c] = __shfl_sync(gmask, fv[c], base);
    }
  }
  // out, emf and nj may each be absent (the per-kernel launch interface
  // asks for fluxes or for the CT face tables alone); the stores are split
  // over the group (component c by lane c mod Q)
  if (out.f[0]) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (c % Q == lane) out.f[c][k] = res[c];
  }
  if (lane == 0 && emf) emf[k] = DIR == 0 ? -res[6] : res[5];
  if (spd) {
    double m = rate;
#pragma unroll
    for (int q = 0; q < Q; ++q) m = fmax(m, __shfl_sync(gmask, rate, base + q));
    if (lane == 0) spd[k] = m;
  }
  if (!nj) return;  // uniform over the block
  // no-jump proof (as in b_face_flux_cs)
  const bool inner = DIR == 0 ? (j0 >= H && j0 + TY - 1 + H < g.ny) : (i0 >= H && i0 + TX - 1 + H < g.nx);
  if (inner) {
    if (lane == 0) nj[k] = flat ? 1 : 0;
    return;
  }
  int proof = 1;
  for (int off = lane - H; off <= H; off += Q) {
    const int mi = face_index(DIR == 0 ? i : i + off, g.nx, g.bc[0], g.bc[1]);
    const int mj = face_index(DIR == 0 ? j + off : j, g.ny, g.bc[2], g.bc[3]);
    const int ti = DIR == 0 ? ((i == g.nx && perx) ? 0 : i) : i + off;
    const int tj = DIR == 0 ? j + off : ((j == g.ny && pery) ? 0 : j);
    if (mi == ti && mj == tj) {
      const int sl = slot(off + H);
      if (!(same[sl >> 5] >> (sl & 31) & 1u)) proof = 0;
      continue;
    }
    if (!in_pad(g, mi, mj)) {
      proof = 0;
      break;
    }
    const long long km = g.idx(mi, mj);
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (!(in.L[c][km] == in.R[c][km])) proof = 0;
  }
  const unsigned nproof = (__ballot_sync(gmask, proof == 0) >> base) & ((1u << Q) - 1u);
  if (lane == 0) nj[k] = nproof == 0 ? 1 : 0;
}

// Component-split recovery (MP7), as described above.
// sm: the caller's shared memory (fq_smem doubles), or null (OWN) where the
// kernel holds only this body and has arrays of its own.
template <int DIR, int ORDER, bool OWN, int TX = kFqTX>
__device__ __forceinline__ void b_face_flux_cs(const Grid& g, const IfaceP& in, const FluxP& out,
                                               double* emf, int* nj, double* spd, double gamma,
                                               const Ctl* ctl, int bx, int by, double* sm) {
  constexpr int H = ORDER == 5 ? 2 : 3, N = 2 * H + 1, Q = ORDER == 5 ? 3 : 4;
  constexpr int FPW = 32 / Q, TY = fq_ty<ORDER>();         // faces per warp, tile rows
  static_assert(4 * FPW == TX * TY, "four warps cover the face tile");
  constexpr int TR = DIR == 0 ? TY + 2 * H : TY;          // tile rows (j)
  constexpr int TC = DIR == 0 ? TX : TX + 2 * H;          // tile columns (i)
  constexpr int PS = fq_plane(TR * TC), FS = fq_face<ORDER>();
  constexpr int kWords = (TR * TC + 31) / 32;
  double* tile;    // component c of slot (row, col): c PS + row TC + col
  unsigned* same;  // staged and L == R in every component: one bit per tile slot
  double* pts;     // per face: Q point rows
  if constexpr (OWN) {
    __shared__ double own_tile[16 * PS];
    __shared__ unsigned own_same[kWords + 1];
    __shared__ __align__(16) double own_pts[4 * FPW * FS];
    tile = own_tile;
    same = own_same;
    pts = own_pts;
  } else {
    tile = sm;
    pts = sm + 16 * PS;
    same = reinterpret_cast<unsigned*>(pts + 4 * FPW * FS);
  }
  if (ctl->status) return;  // uniform over the block
  const int i0 = bx * TX, j0 = by * TY;
  const bool perx = g.bc[0] == 0 && g.bc[1] == 0, pery = g.bc[2] == 0 && g.bc[3] == 0;
  static_assert(TR * TC <= kFqThreads, "one tile slot per thread");
  {
    const int e = threadIdx.x;
    const int row = e / TC, col = e - row * TC;
    int fi, fj;
    bool valid;
    if (DIR == 0) {
      const int ii = i0 + col;
      fi = (ii == g.nx && perx) ? 0 : ii;
      fj = j0 - H + row;
      valid = e < TR * TC && ii <= g.nx && fj >= -g.ng && fj < g.ny + g.ng;
    } else {
      const int jj = j0 + row;
      fj = (jj == g.ny && pery) ? 0 : jj;
      fi = i0 - H + col;
      valid = e < TR * TC && jj <= g.ny && fi >= -g.ng && fi < g.nx + g.ng;
    }
    const long long kk = valid ? g.idx(fi, fj) : 0;
    bool eq = valid;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double a = valid ? __ldg(in.L[c] + kk) : 0.0;
      const double b = valid ? __ldg(in.R[c] + kk) : 0.0;
      if (e < TR * TC) {
        tile[c * PS + e] = a;
        tile[(8 + c) * PS + e] = b;
      }
      eq = eq && a == b;
    }
    const unsigned w = __ballot_sync(0xffffffffu, eq);
    if ((e & 31) == 0 && e / 32 < kWords) same[e / 32] = w;
    if (e == 0) same[kWords] = 0u;
  }
  __syncthreads();
  const bool inner = DIR == 0 ? (j0 >= H && j0 + TY - 1 + H < g.ny) : (i0 >= H && i0 + TX - 1 + H < g.nx);
  // no slot with a jump (block-uniform; the first word stops a developed flow)
  if (same[0] == ~0u && inner && stencil_words<TR * TC>(same)) {
    bool one = true;
    if (threadIdx.x < TR * TC) {
#pragma unroll
      for (int c = 0; c < 8; ++c) one = one && tile[c * PS + threadIdx.x] == tile[c * PS];
    }
    if (__syncthreads_and(one)) {
      constant_tile_flux<DIR, ORDER, TX>(g, out, emf, nj, spd, gamma, i0, j0,
                                         [&](int c) { return tile[c * PS]; });
      return;
    }
  }
  constexpr bool kLF = false;
  const int wl = threadIdx.x & 31;
  static_assert(FPW * Q == 32, "every lane has a group");
  const int lane = wl % Q, base = wl - lane;
  const unsigned gmask = ((1u << Q) - 1u) << base;
  const int face = (threadIdx.x >> 5) * FPW + wl / Q;
  const int fx = face % TX, fy = face / TX;
  const int i = i0 + fx, j = j0 + fy;
  if (i > g.nx || j > g.ny) return;  // whole groups leave together
  const long long k = g.idx(i, j);
  const double h = DIR == 0 ? g.dx : g.dy;
  // tile slot of stencil tap t (t = H is the face itself)
  auto slot = [&](int t) { return DIR == 0 ? (fy + t) * TC + fx : fy * TC + fx + t; };
  double* const fp = pts + face * FS;  // this face's point rows
  const bool flat = stencil_flat<DIR, N>(same, slot(0), TC);
  // point values of components lane, lane + Q, ... at the Q Gauss nodes
#pragma unroll
  for (int m = 0; m < (16 + Q - 1) / Q; ++m) {
    const int c = lane + Q * m;
    if (c < 16) {
      double s[N], v[Q];
#pragma unroll
      for (int t = 0; t < N; ++t) s[t] = tile[c * PS + slot(t)];
      point_values<ORDER>(s, v);
#pragma unroll
      for (int p = 0; p < Q; ++p) fp[p * kFqRow + c] = v[p];
    }
  }
  __syncwarp(gmask);
  St l, r;
  {
    const double2* row = reinterpret_cast<const double2*>(fp + lane * kFqRow);
    const double2 a0 = row[0], a1 = row[1], a2 = row[2], a3 = row[3];
    const double2 b0 = row[4], b1 = row[5], b2 = row[6], b3 = row[7];
    l = St{a0.x, a0.y, a1.x, a1.y, a2.x, a2.y, a3.x, a3.y};
    r = St{b0.x, b0.y, b1.x, b1.y, b2.x, b2.y, b3.x, b3.y};
  }
  double irl = rcp_nr(l.rho), irr = rcp_nr(r.rho);
  double prl = pressure_f(l, gamma, irl), prr = pressure_f(r, gamma, irr);
  const bool ok = point_admissible_p(l, prl) && point_admissible_p(r, prr);
  auto centre = [&](bool left) {
    const int o = left ? 0 : 8, sc = slot(H);
    return St{tile[o * PS + sc],       tile[(o + 1) * PS + sc], tile[(o + 2) * PS + sc],
              tile[(o + 3) * PS + sc], tile[(o + 4) * PS + sc], tile[(o + 5) * PS + sc],
              tile[(o + 6) * PS + sc], tile[(o + 7) * PS + sc]};
  };
  const unsigned bad = (__ballot_sync(gmask, !ok) >> base) & ((1u << Q) - 1u);
  const bool group_ok = bad == 0;
  const int first_bad = bad ? __ffs(bad) - 1 : Q;
  double rate = 0.0;
  if (spd) {
    if (lane == 0) {
      const St a = centre(true), b = centre(false);
      rate = face_rate<DIR, ORDER>(a, b, gamma, h, rcp_rho(a.rho), rcp_rho(b.rho));
    }
    if (lane < first_bad) rate = fmax(rate, face_rate<DIR, ORDER>(l, r, gamma, h, irl, irr));
  }
  const bool solve = group_ok || lane == 0;
  if (!group_ok) {
    l = centre(true);
    r = centre(false);
    irl = rcp_rho(l.rho);
    irr = rcp_rho(r.rho);
    prl = pressure_f(l, gamma, irl);
    prr = pressure_f(r, gamma, irr);
  }
  double fv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (solve) {
    const Fx f = flat ? flat_flux<DIR>(l, prl, irl) : riemann<DIR, false>(l, r, kLF, gamma, irl, irr, prl, prr);
    fv[0] = f.rho; fv[1] = f.mx; fv[2] = f.my; fv[3] = f.mz;
    fv[4] = f.E;   fv[5] = f.bx; fv[6] = f.by; fv[7] = f.bz;
  }
  // the point fluxes replace the lane's own point row (no other lane reads
  // it after the exchange above)
  {
    double2* row = reinterpret_cast<double2*>(fp + lane * kFqRow);
    row[0] = make_double2(fv[0], fv[1]);
    row[1] = make_double2(fv[2], fv[3]);
    row[2] = make_double2(fv[4], fv[5]);
    row[3] = make_double2(fv[6], fv[7]);
  }
  __syncwarp(gmask);
  // Gauss sums of components lane, lane + Q, ... in node order (or lane 0's
  // single solve at the face state when a point was not admissible)
  constexpr int RC = (8 + Q - 1) / Q;
  double res[RC];
#pragma unroll
  for (int m = 0; m < RC; ++m) {
    const int c = lane + Q * m;
    res[m] = 0.0;
    if (c < 8) {
      if (group_ok) {
        double sq[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) sq[q] = fp[q * kFqRow + c];
        res[m] = gauss_avg<ORDER>(sq);
      } else {
        res[m] = fp[c];
      }
    }
  }
  // out, emf and nj may each be absent (the per-kernel launch interface
  // asks for fluxes or for the CT face tables alone)
  if (out.f[0]) {
#pragma unroll
    for (int m = 0; m < RC; ++m)
      if (lane + Q * m < 8) out.f[lane + Q * m][k] = res[m];
  }
  // face E_z = -F(by) of an x face, F(bx) of a y face: the lane holding it
  constexpr int EC = DIR == 0 ? 6 : 5;
  if (emf && lane == EC % Q) emf[k] = DIR == 0 ? -res[EC / Q] : res[EC / Q];
  if (spd) {
    double m = rate;
#pragma unroll
    for (int q = 0; q < Q; ++q) m = fmax(m, __shfl_sync(gmask, rate, base + q));
    if (lane == 0) spd[k] = m;
  }
  if (!nj) return;  // uniform over the block
  // no-jump proof over the 2H+1 transverse taps (mapped like every CT table
  // read).  Where no tap of the tile is mapped, the staged bits are the proof
  // (a block-uniform test; the general form below is about 100 instructions).
  if (inner) {
    if (lane == 0) nj[k] = flat ? 1 : 0;
    return;
  }
  // the group splits the taps; one whose mapped face is the one staged in its
  // tile slot reads the staged bit, the others read memory
  int proof = 1;
  for (int off = lane - H; off <= H; off += Q) {
    const int mi = face_index(DIR == 0 ? i : i + off, g.nx, g.bc[0], g.bc[1]);
    const int mj = face_index(DIR == 0 ? j + off : j, g.ny, g.bc[2], g.bc[3]);
    const int ti = DIR == 0 ? ((i == g.nx && perx) ? 0 : i) : i + off;
    const int tj = DIR == 0 ? j + off : ((j == g.ny && pery) ? 0 : j);
    if (mi == ti && mj == tj) {
      const int sl = slot(off + H);
      if (!(same[sl >> 5] >> (sl & 31) & 1u)) proof = 0;
      continue;
    }
    if (!in_pad(g, mi, mj)) {
      proof = 0;
      break;
    }
    const long long km = g.idx(mi, mj);
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (!(in.L[c][km] == in.R[c][km])) proof = 0;
  }
  const unsigned nproof = (__ballot_sync(gmask, proof == 0) >> base) & ((1u << Q) - 1u);
  if (lane == 0) nj[k] = nproof == 0 ? 1 : 0;
}

// Shared memory (doubles) of one direction's tile, point rows and bits.
template <int DIR, int ORDER>
constexpr int fq_smem() {
  constexpr int H = ORDER == 5 ? 2 : 3, TY = fq_ty<ORDER>();
  constexpr int cells = DIR == 0 ? (TY + 2 * H) * kFqTX : TY * (kFqTX + 2 * H), bits = 4;
  if (ORDER == 5) return 16 * cells + bits;
  return 16 * fq_plane(cells) + 32 * fq_face<ORDER>() + bits;
}
template <int ORDER>
constexpr int fq_smem_both() {
  return fq_smem<0, ORDER>() > fq_smem<1, ORDER>() ? fq_smem<0, ORDER>() : fq_smem<1, ORDER>();
}
// TX: faces per tile row; the block is four warps of 32 / Q groups each.
template <int DIR, int ORDER, bool OWN, int TX = kFqTX>
__device__ __forceinline__ void b_face_flux_qs(const Grid& g, const IfaceP& in, const FluxP& out,
                                               double* emf, int* nj, double* spd, double gamma,
                                               const Ctl* ctl, int bx, int by, double* sm) {
  if constexpr (ORDER == 7)
    b_face_flux_cs<DIR, ORDER, OWN, TX>(g, in, out, emf, nj, spd, gamma, ctl, bx, by, sm);
  else
    b_face_flux_pt<DIR, ORDER, TX>(g, in, out, emf, nj, spd, gamma, ctl, bx, by, sm);
}

// Outputs of one direction's face flux.
struct FaceOut {
  FluxP f;
  double* emf;
  int* nj;
  double* spd;
};
// One direction per launch, for MP7 grids beyond kFqPairBlocks.
template <int DIR, int ORDER>
__global__ void __launch_bounds__(kFqThreads, kFqBlocksPerSm)
    k_face_flux_one(Grid g, IfaceP in, FluxP out, double* emf, int* nj, double* spd, double gamma,
                    const Ctl* ctl) {
  b_face_flux_qs<DIR, ORDER, true, kFqTX>(g, in, out, emf, nj, spd, gamma, ctl, blockIdx.x,
                                          blockIdx.y, nullptr);
}
// One direction (dir0 + blockIdx.z) or both, as k_reconstruct.  At MP5 the
// pair is faster at every size (1024^2: 1.35 -> 1.32 ms per step).  At MP7 the
// kernel that holds both bodies is slower where the grid fills the chip many
// times over (1024^2: 1.38 -> 1.51) and faster where it does not (64^2: 0.060 ->
// 0.042, 200 x 150, 988 blocks a direction: 0.086 -> 0.075): the line is two
// waves of resident blocks.
constexpr long long kFqPairBlocks = 2 * 148 * kFqBlocksPerSm;
template <int ORDER>
__global__ void __launch_bounds__(kFqThreads, kFqBlocksPerSm)
    k_face_flux_qs(Grid g, IfaceP ix, IfaceP iy, FaceOut ox, FaceOut oy, double gamma,
                   const Ctl* ctl, int dir0) {
  __shared__ __align__(16) double sm[fq_smem_both<ORDER>()];
  if (dir0 + int(blockIdx.z) == 0)
    b_face_flux_qs<0, ORDER, false, kFqTX>(g, ix, ox.f, ox.emf, ox.nj, ox.spd, gamma, ctl, blockIdx.x,
                                    blockIdx.y, sm);
  else
    b_face_flux_qs<1, ORDER, false, kFqTX>(g, iy, oy.f, oy.emf, oy.nj, oy.spd, gamma, ctl, blockIdx.x,
                                    blockIdx.y, sm);
}

}  // namespace

// ===========================================================================
// Constrained transport and the stage update
// ===========================================================================
namespace {

// E_z = -(v x B)_z (mhd_ct.hip:408-417, zero background)
// E_z = -(v x B)_z from the state and its 1/rho (one reciprocal shared with
// the point's admissibility test instead of a division per velocity
// component: a rounding-level difference)
__device__ __forceinline__ double physical_ez_ir(const St& s, double ir) {
  const double vx = s.mx * ir, vy = s.my * ir;
  return __dadd_rn(__dmul_rn(vy, s.bx), __dmul_rn(vx, -s.by));
}
__device__ __forceinline__ double physical_ez(const St& s) { return physical_ez_ir(s, 1.0 / s.rho); }

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Orders 1 and 2: E_z of the cell states (mhd_ct.hip:457-629); on stage 0 also
// the CFL max-reduction over cells (mhd_reduce.hip:418-501): warp shuffles, one
// atomic per block.
template <int ORDER>
__global__ void __launch_bounds__(128) k_cell_emf(Grid g, StateP u, double* cell_ez,
                                                  const double* xs, const double* ys,
                                                  int cfl_reduce, Ctl* ctl) {
  __shared__ int s_stop;
  __shared__ double s_max[4];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  if (tid == 0) s_stop = ctl->status;
  __syncthreads();
  if (s_stop) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const bool phx = g.bc[1] != 0, phy = g.bc[3] != 0;
  if (i <= g.nx && j <= g.ny && !((i == g.nx && !phx) || (j == g.ny && !phy))) {
    const long long k = g.idx(i, j);
    const St c0 = ORDER <= 1 ? load_cell1(u, g, i, j) : load_cell(u, k);
    cell_ez[k] = physical_ez(c0);
  }
  if (!cfl_reduce) return;
  double local = 0.0;
  if (i < g.nx && j < g.ny && g.in_window(i, j)) {
    const long long k = g.idx(i, j);
    const double r = (xs[k] + xs[k + 1]) + (ys[k] + ys[k + g.pitch]);
    local = isfinite(r) ? fmax(0.0, r) : kInf;
  }
  local = warp_max(local);
  if ((tid & 31) == 0) s_max[tid >> 5] = local;
  __syncthreads();
  if (tid == 0) {
    double m = s_max[0];
    for (int w = 1; w < (int)(blockDim.x * blockDim.y + 31) / 32; ++w) m = fmax(m, s_max[w]);
    atomicMax(&ctl->max_rate, dbits(m));
  }
}

// Tiled form of k_cell_emf for MP5/MP7: a 16x16 tile of cells and its
// H-wide halo are staged in shared memory once; for each x-node the
// x-recovered rows of the tile (all 8 components) are formed once in shared
// memory and every cell then recovers its y-nodes from them.  Same sums in
// the same order as k_cell_emf.  A square tile recovers fewer halo rows per
// cell than 32x8 (22/16 against 14/8 at MP7).
constexpr int kCellTX = 16, kCellTY = 16;

// TMA staging of the tile: rows of kTmaBW doubles (192 bytes) starting one
// cell left of the stencil's first column, so that the innermost coordinate
// of every copy is even (16-byte aligned); planes of SY rows are multiples of
// 128 bytes at both orders.
constexpr int kTmaBW = 24;

template <int ORDER, bool TMA = false>
constexpr int cell_smem_doubles() {
  constexpr int H = ORDER == 7 ? 3 : 2, SY = kCellTY + 2 * H;
  // TMA: 16 more doubles so that the staged planes can start on 128 bytes
  return 8 * SY * (TMA ? kTmaBW : kCellTX + 2 * H) + 8 * SY * kCellTX + (TMA ? 16 : 0);
}

// 3-D tiled TMA load of one box into shared memory, completing on `bar`.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y,
                                            int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(tc::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(tc::smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

// TMA: the eight state planes of the tile come in by one TMA copy each
// (issued by one thread, completing on an mbarrier whose wait is bounded)
// from `map`, the register's 3-D tensor map; out-of-range cells are filled
// with zeros by the copy, as the plain staging does.
template <int ORDER, bool TMA = false>
__device__ __forceinline__ void b_cell_emf_s(const Grid& g, const StateP& u, double* cell_ez,
                                             const double* xs, const double* ys, int cfl_reduce,
                                             double gamma, Ctl* ctl, int bx, int by,
                                             const CUtensorMap* map = nullptr) {
  constexpr int H = ORDER == 7 ? 3 : 2, N = 2 * H + 1, Q = ORDER == 7 ? 4 : 3;
  constexpr int TX = kCellTX, TY = kCellTY, SX = TX + 2 * H, SY = TY + 2 * H;
  // row stride and column offset of the staged tile: S[c][r][x] is the
  // stencil cell (i0 - H + x, j0 - H + r) at S + (c * SY + r) * RS + XO + x
  constexpr int RS = TMA ? kTmaBW : SX, XO = TMA ? 1 : 0;
  static_assert(!TMA || (SX + XO <= kTmaBW && (SY * kTmaBW * 8) % 128 == 0), "TMA box");
  extern __shared__ __align__(128) double sm[];
  // TMA destinations start on 128 bytes; the offset is taken inside the
  // shared array, so that the compiler keeps shared-memory loads (a pointer
  // rounded as an integer is generic: the cell EMF phase took 7.6 instead
  // of 7.1 ms per rotor 4096^2 MP7 step)
  double* S = TMA ? sm + ((128u - (tc::smem_u32(sm) & 127u)) & 127u) / sizeof(double)
                  : sm;          // [8][SY][RS] staged state
  double* X = S + 8 * SY * RS;  // [8][SY][TX] x-recovered rows of one x-node
  __shared__ int s_stop;
  __shared__ double s_max[8];
  __shared__ uint64_t s_bar;
  const int tid = threadIdx.y * TX + threadIdx.x;
  if (tid == 0) s_stop = ctl->status;
  __syncthreads();
  if (s_stop) return;
  const int i0 = bx * TX, j0 = by * TY;
  const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
  if constexpr (TMA) {
    // padded coordinates: x0 = i0 - H + ng - XO is even because ng - H = 1
    // at both orders and i0 is a multiple of 16
    if (tid == 0) {
      tc::mbar_init(&s_bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(&s_bar, uint32_t(8 * SY * kTmaBW * sizeof(double)));
      const int x0 = i0 - H + g.ng - XO, y0 = j0 - H + g.ng;
      constexpr int kZ[8] = {0, 1, 2, 3, 4, 8, 9, 7};  // rho..E, bxc, byc, bz
#pragma unroll
      for (int c = 0; c < 8; ++c) tma_load_3d(S + c * SY * kTmaBW, map, x0, y0, kZ[c], &s_bar);
    }
    __syncthreads();  // the barrier is initialised before anyone waits on it
    // one warp polls the mbarrier; the others sleep in the block barrier,
    // which also orders the landed tile before their reads
    bool arrived = true;
    if (tid < 32) arrived = tc::mbar_wait(&s_bar, 0);
    if (!__syncthreads_and(arrived ? 1 : 0)) {
      // the copies did not land in time: report it, give them a second
      // bounded wait so that none is still writing when the block exits
      if (tid == 0) {
        atomicOr(&ctl->status, kStatusWaitExpired);
        tc::mbar_wait(&s_bar, 0);
      }
      __syncthreads();
      return;
    }
  } else {
  // staging: one index computation per staged cell, its 8 components
  // loaded with the same offset
  for (int r = threadIdx.y; r < SY; r += TY) {
    for (int x = threadIdx.x; x < SX; x += TX) {
      const int ii = i0 - H + x, jj = j0 - H + r;
      const bool in = in_pad(g, ii, jj);
      const long long kk = in ? g.idx(ii, jj) : 0;
      double* dst = S + r * SX + x;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const double* src = c < 5 ? u.c[c] : c == 5 ? u.bxc : c == 6 ? u.byc : u.c[7];
        dst[c * SY * SX] = in ? __ldg(src + kk) : 0.0;
      }
    }
  }
  __syncthreads();
  }
  const bool phx = g.bc[1] != 0, phy = g.bc[3] != 0;
  const bool active =
      i <= g.nx && j <= g.ny && !((i == g.nx && !phx) || (j == g.ny && !phy));
  // a tile of one state (uniform gas): its E_z is that state's.  Tested on the
  // density of the tile's own cells first, where any other tile stops.  Rotor
  // 4096^2 MP7: 7.4 -> 1.7 ms per step.
  bool uniform;
  {
    auto at = [&](int c, int r, int x) { return S[(c * SY + r) * RS + XO + x]; };
    uniform = __syncthreads_and(at(0, threadIdx.y + H, threadIdx.x + H) == at(0, 0, 0));
    if (uniform) {
      bool one = true;
      for (int t = tid; t < SY * SX; t += TX * TY) {
        const int r = t / SX, x = t - r * SX;
#pragma unroll
        for (int c = 0; c < 8; ++c) one = one && at(c, r, x) == at(c, 0, 0);
      }
      uniform = __syncthreads_and(one);
    }
  }
  double pt[Q][Q];
  bool ok = !uniform;
  if (!uniform)
#pragma unroll
  for (int qx = 0; qx < Q; ++qx) {
    double wx[N];
#pragma unroll
    for (int t = 0; t < N; ++t) wx[t] = point_w<ORDER>(qx, t);
    // x-recovery of every staged row (component c, row r) at this x node:
    // task = (row t = c * SY + r, column pair p); the two outputs' N + 1
    // taps come in as 16-byte loads (the staged rows start on 16 bytes;
    // with XO = 1 the pair's taps start one double into the first load)
    static_assert(RS % 2 == 0 && TX % 2 == 0, "16-byte rows");
    constexpr int NL = (XO + N + 2) / 2;  // 16-byte loads per pair
    for (int tk = tid; tk < 8 * SY * (TX / 2); tk += TX * TY) {
      const int t = tk / (TX / 2), pr = tk - t * (TX / 2);
      const double2* row = reinterpret_cast<const double2*>(S + t * RS + 2 * pr);
      double v[2 * NL];
#pragma unroll
      for (int q = 0; q < NL; ++q) {
        const double2 d = row[q];
        v[2 * q] = d.x;
        v[2 * q + 1] = d.y;
      }
      double s0[N], s1[N];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        s0[q] = v[XO + q];
        s1[q] = v[XO + 1 + q];
      }
      reinterpret_cast<double2*>(X + t * TX)[pr] = make_double2(wsum<N>(wx, s0), wsum<N>(wx, s1));
    }
    __syncthreads();
    if (active && ok) {
      double st[Q][8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        double smp[N];
#pragma unroll
        for (int t = 0; t < N; ++t) smp[t] = X[(c * SY + threadIdx.y + t) * TX + threadIdx.x];
        double pv[Q];
        point_values<ORDER>(smp, pv);
#pragma unroll
        for (int qy = 0; qy < Q; ++qy) st[qy][c] = pv[qy];
      }
#pragma unroll
      for (int qy = 0; qy < Q; ++qy) {
        const St p{st[qy][0], st[qy][1], st[qy][2], st[qy][3],
                   st[qy][4], st[qy][5], st[qy][6], st[qy][7]};
        const double ir = 1.0 / p.rho;
        if (!point_admissible_ir(p, gamma, ir)) ok = false;
        pt[qy][qx] = physical_ez_ir(p, ir);
      }
    }
    __syncthreads();
  }
  if (active) {
    const long long k = g.idx(i, j);
    double e;
    if (ok) {
      double row[Q];
#pragma unroll
      for (int qy = 0; qy < Q; ++qy) row[qy] = gauss_avg<ORDER>(pt[qy]);
      e = gauss_avg<ORDER>(row);
    } else if (uniform) {
      // what its points give, bit for bit: the same correctly rounded 1 / rho,
      // whether they are admissible or not; the staged state, not the register's
      auto at = [&](int c) { return S[c * SY * RS + XO]; };
      e = physical_ez(St{at(0), at(1), at(2), at(3), at(4), at(5), at(6), at(7)});
    } else {
      e = physical_ez(load_cell(u, k));
    }
    cell_ez[k] = e;
  }
  if (!cfl_reduce) return;
  double local = 0.0;
  if (i < g.nx && j < g.ny && g.in_window(i, j)) {
    const long long k = g.idx(i, j);
    const double r = (xs[k] + xs[k + 1]) + (ys[k] + ys[k + g.pitch]);
    local = isfinite(r) ? fmax(0.0, r) : kInf;
  }
  local = warp_max(local);
  if ((tid & 31) == 0) s_max[tid >> 5] = local;
  __syncthreads();
  if (tid == 0) {
    double m = s_max[0];
    for (int w = 1; w < 8; ++w) m = fmax(m, s_max[w]);
    atomicMax(&ctl->max_rate, dbits(m));
  }
}

template <int ORDER>
__global__ void __launch_bounds__(256, 3) k_cell_emf_s(Grid g, StateP u, double* cell_ez,
                                                    const double* xs, const double* ys,
                                                    int cfl_reduce, double gamma, Ctl* ctl) {
  b_cell_emf_s<ORDER>(g, u, cell_ez, xs, ys, cfl_reduce, gamma, ctl, blockIdx.x, blockIdx.y);
}

// The same with the tile staged by TMA from the register's tensor map
// (single-instance path; this GPU's own memory, no multicast).
template <int ORDER>
__global__ void __launch_bounds__(256, 3) k_cell_emf_tma(Grid g, StateP u,
                                                      const __grid_constant__ CUtensorMap map,
                                                      double* cell_ez, const double* xs,
                                                      const double* ys, int cfl_reduce,
                                                      double gamma, Ctl* ctl) {
  b_cell_emf_s<ORDER, true>(g, u, cell_ez, xs, ys, cfl_reduce, gamma, ctl, blockIdx.x,
                            blockIdx.y, &map);
}

// Face -> edge interpolation (mhd_ct.hip:50-97) as a sample plus weighted
// differences from it, so that equal samples return their value (the
// reference's constant shortcut); *cst, where asked for, is whether they are.
template <int NT>
__device__ __forceinline__ double edge_interp(const double* e, bool* cst = nullptr) {
  if (NT == 2) {
    if (cst) *cst = e[0] == e[1];
    return __dmul_rn(__dadd_rn(e[0], e[1]), 0.5);  // = / 2 exactly
  }
  double d[NT];
  unsigned bits = 0u;
#pragma unroll
  for (int q = 1; q < NT; ++q) {
    d[q] = __dsub_rn(e[q], e[0]);
    // a zero of either sign only where finite samples are equal
    bits |= (unsigned(__double2hiint(d[q])) & 0x7fffffffu) | unsigned(__double2loint(d[q]));
  }
  double r;
  if (NT == 6)
    r = fma(1.0 / 60.0, fma(37.0, d[2] + d[3], fma(-8.0, d[1] + d[4], d[5])), e[0]);
  else
    r = fma(1.0 / 840.0,
            fma(533.0, d[3] + d[4], -139.0 * (d[2] + d[5])) + fma(29.0, d[1] + d[6], -3.0 * d[7]),
            e[0]);
  bool same = bits == 0u;
  if (r != r) {  // equal infinities differ by NaN and return their value
    same = true;
#pragma unroll
    for (int q = 1; q < NT; ++q) same = same && e[q] == e[0];
    if (same) r = e[0];
  }
  if (cst) *cst = same;
  return r;
}

// Upwind CT corner E_z = ex + ey - centred, with the exact one-dimensional
// limits (mhd_ct.hip:811-878).
template <int ORDER>
__global__ void __launch_bounds__(128) k_corner_emf(Grid g, const double* cell_ez,
                                                    const double* xemf, const double* yemf,
                                                    const int* xnj, const int* ynj, double* ez,
                                                    const Ctl* ctl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i > g.nx || j > g.ny) return;
  if (ctl->status) return;
  const long long k = g.idx(i, j);
  const bool conducting = (i == 0 && g.bc[0] == 2) || (i == g.nx && g.bc[1] == 2) ||
                          (j == 0 && g.bc[2] == 2) || (j == g.ny && g.bc[3] == 2);
  if (conducting) {
    ez[k] = 0.0;
    return;
  }
  constexpr int LO = ORDER >= 7 ? -4 : ORDER >= 5 ? -3 : -1;
  constexpr int NT = ORDER >= 7 ? 8 : ORDER >= 5 ? 6 : 2;
  int mi[NT], mj[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    mi[q] = face_index(i + LO + q, g.nx, g.bc[0], g.bc[1]);
    mj[q] = face_index(j + LO + q, g.ny, g.bc[2], g.bc[3]);
  }
  const int fi = face_index(i, g.nx, g.bc[0], g.bc[1]);
  const int fj = face_index(j, g.ny, g.bc[2], g.bc[3]);
  double e[NT], line[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) e[q] = xemf[g.idx(fi, mj[q])];
  const double ex = edge_interp<NT>(e);
#pragma unroll
  for (int q = 0; q < NT; ++q) e[q] = yemf[g.idx(mi[q], fj)];
  const double ey = edge_interp<NT>(e);
  // cell-centred reference, and the constancy of the cell table along x
  // (y_only) and along y (x_only) over the same stencil
  bool const_x = true, const_y = true;
  double col0[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    double c[NT];
#pragma unroll
    for (int p = 0; p < NT; ++p) c[p] = cell_ez[g.idx(mi[p], mj[q])];
#pragma unroll
    for (int p = 1; p < NT; ++p) const_x = const_x && (c[p] == c[0]);
    if (q == 0) {
#pragma unroll
      for (int p = 0; p < NT; ++p) col0[p] = c[p];
    } else {
#pragma unroll
      for (int p = 0; p < NT; ++p) const_y = const_y && (c[p] == col0[p]);
    }
    line[q] = edge_interp<NT>(c);
  }
  const double centred = edge_interp<NT>(line);
  bool nj_y = true, nj_x = true;
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    const int a = mi[q], b = mj[q];
    nj_y = nj_y && in_pad(g, a, fj) && ynj[g.idx(a, fj)] != 0;
    nj_x = nj_x && in_pad(g, fi, b) && xnj[g.idx(fi, b)] != 0;
  }
  const bool x_only = nj_y && const_y;
  const bool y_only = nj_x && const_x;
  double v;
  if (x_only && !y_only) v = ex;
  else if (y_only && !x_only) v = ey;
  else v = crsum3(ex, ey, -centred);
  ez[k] = v;
}

// Same corner EMF for a tile of 32 x 16 corners (32 x 8 threads, two rows
// each) with its tables staged in shared memory: the mapped cell E_z, the
// x-face E_z and proofs of its corner columns, the y-face ones of its corner
// rows.  The centred value is separable: each staged row's x-interpolation
// at the 32 corner columns (xr) and whether the row is constant over that
// stencil (xc), and whether each staged column is constant over the corner
// rows' y-stencils (yc), are formed once per tile.  Bound by the instructions
// of the staging and its redundant halo: 16 rows stage 1.4 cell rows a corner
// row against 2.75 for four, and a tile whose taps are all inside the tables
// (a block-uniform test) skips the index mapping (flow 2048^2 MP7: 0.571 -> 0.413 ms
// per step).
constexpr int kCornerTY = 16;
template <int ORDER>
__device__ __forceinline__ void b_corner_emf_s(const Grid& g, const double* cell_ez, const double* xemf,
                                               const double* yemf, const int* xnj, const int* ynj,
                                               double* ez, const Ctl* ctl, int bx, int by) {
  constexpr int LO = ORDER >= 7 ? -4 : ORDER >= 5 ? -3 : -1;
  constexpr int NT = ORDER >= 7 ? 8 : ORDER >= 5 ? 6 : 2;
  constexpr int TY = kCornerTY, TW = 32 + NT - 1, TH = TY + NT - 1;
  __shared__ double tile[TH][TW];
  __shared__ double sxe[TH][32], sye[TY][TW];
  __shared__ double xr[TH][32];
  __shared__ unsigned char sxn[TH][32], syn[TY][TW], xc[TH][32], yc[TY][TW];
  if (ctl->status) return;  // uniform over the block
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i0 = bx * 32, j0 = by * TY;
  // taps reach LO .. LO + NT - 1 about every corner of the tile; inside
  // [0, n) no axis maps them
  const bool inner = i0 + LO >= 0 && i0 + 31 + LO + NT - 1 < g.nx && j0 + LO >= 0 &&
                     j0 + TY - 1 + LO + NT - 1 < g.ny;
  auto mapx = [&](int q) { return inner ? q : face_index(q, g.nx, g.bc[0], g.bc[1]); };
  auto mapy = [&](int q) { return inner ? q : face_index(q, g.ny, g.bc[2], g.bc[3]); };
  // column tx (and the NT - 1 beyond 32) of every row by the warp's row ty
#pragma unroll
  for (int b = ty; b < TH; b += 8) {
    const int mj = mapy(j0 + LO + b);
    const long long row = g.idx(0, mj);
    tile[b][tx] = __ldg(cell_ez + row + mapx(i0 + LO + tx));
    if (tx < NT - 1) tile[b][32 + tx] = __ldg(cell_ez + row + mapx(i0 + LO + 32 + tx));
    const int fi = mapx(i0 + tx);
    sxe[b][tx] = __ldg(xemf + row + fi);
    sxn[b][tx] = __ldg(xnj + row + fi) != 0;
  }
#pragma unroll
  for (int b = ty; b < TY; b += 8) {
    const int fj = mapy(j0 + b);
    const long long row = g.idx(0, fj);
    const int mi = mapx(i0 + LO + tx);
    sye[b][tx] = __ldg(yemf + row + mi);
    syn[b][tx] = __ldg(ynj + row + mi) != 0;
    if (tx < NT - 1) {
      const int m2 = mapx(i0 + LO + 32 + tx);
      sye[b][32 + tx] = __ldg(yemf + row + m2);
      syn[b][32 + tx] = __ldg(ynj + row + m2) != 0;
    }
  }
  __syncthreads();
  for (int b = ty; b < TH; b += 8) {
    double c[NT];
    bool cst;
#pragma unroll
    for (int p = 0; p < NT; ++p) c[p] = tile[b][tx + p];
    xr[b][tx] = edge_interp<NT>(c, &cst);
    xc[b][tx] = cst;
  }
  auto column = [&](int b, int a) {
    const double c0 = tile[b][a];
    bool cst = true;
#pragma unroll
    for (int q = 1; q < NT; ++q) cst = cst && (tile[b + q][a] == c0);
    yc[b][a] = cst;
  };
  for (int b = ty; b < TY; b += 8) {
    column(b, tx);
    if (tx < NT - 1) column(b, 32 + tx);
  }
  __syncthreads();
  const int i = i0 + tx;
  if (i > g.nx) return;
#pragma unroll 1
  for (int r = ty; r < TY; r += 8) {
    const int j = j0 + r;
    if (j > g.ny) return;
    const long long k = g.idx(i, j);
    const bool conducting = (i == 0 && g.bc[0] == 2) || (i == g.nx && g.bc[1] == 2) ||
                            (j == 0 && g.bc[2] == 2) || (j == g.ny && g.bc[3] == 2);
    if (conducting) {
      ez[k] = 0.0;
      continue;
    }
    double e[NT];
    unsigned only_y = 1u, only_x = 1u;  // no x jump and rows constant; no y jump and columns constant
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      e[q] = sxe[r + q][tx];
      only_y &= unsigned(sxn[r + q][tx]) & unsigned(xc[r + q][tx]);
    }
    const double ex = edge_interp<NT>(e);
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      e[q] = sye[r][tx + q];
      only_x &= unsigned(syn[r][tx + q]) & unsigned(yc[r][tx + q]);
    }
    const double ey = edge_interp<NT>(e);
#pragma unroll
    for (int q = 0; q < NT; ++q) e[q] = xr[r + q][tx];
    const double centred = edge_interp<NT>(e);
    ez[k] = only_x == only_y ? crsum3(ex, ey, -centred) : only_x ? ex : ey;
  }
}

template <int ORDER>
__global__ void __launch_bounds__(256, 4) k_corner_emf_s(Grid g, const double* cell_ez,
                                                      const double* xemf, const double* yemf,
                                                      const int* xnj, const int* ynj, double* ez,
                                                      const Ctl* ctl) {
  b_corner_emf_s<ORDER>(g, cell_ez, xemf, yemf, xnj, ynj, ez, ctl, blockIdx.x, blockIdx.y);
}

// Flux difference + EMF curl + Shu-Osher combine (mhd_update.hip:21-206,
// mhd_ct.hip:893-931, mhd_solver.cpp:840-874).  Writes cells and the owned
// high faces of the output; ghosts are closed by fill_ghosts afterwards.
__device__ __forceinline__ void b_update(const Grid& g, const StateP& un, const StateP& us,
                                         const StateP& out, const FluxP& fx, const FluxP& fy,
                                         const double* ez, const double* dt_dev, double dt_host,
                                         int stage, const Ctl* ctl, int bx, int by) {
  const int i = bx * blockDim.x + threadIdx.x;
  const int j = by * blockDim.y + threadIdx.y;
  if (i > g.nx || j > g.ny) return;
  if (ctl->status) return;
  const double dt = dt_dev ? *dt_dev : dt_host;
  double a, b, c;
  if (stage == 0) {
    a = 1.0; b = 0.0; c = dt;
  } else if (stage == 1) {
    a = 3.0 / 4.0; b = 1.0 / 4.0; c = (1.0 / 4.0) * dt;
  } else {
    a = 1.0 / 3.0; b = 2.0 / 3.0; c = (2.0 / 3.0) * dt;
  }
  auto combine = [&](double vn, double vs, double d) {
    // rk_weighted_sum (mhd_update.hip:113-135): zero weights skip operands
    if (b == 0.0) return __dadd_rn(__dmul_rn(a, vn), __dmul_rn(c, d));
    return crsum3(__dmul_rn(a, vn), __dmul_rn(b, vs), __dmul_rn(c, d));
  };
  const long long k = g.idx(i, j);
  const double rdx = pow2_recip(g.dx), rdy = pow2_recip(g.dy);
  if (i < g.nx && j < g.ny) {
    const int cc[6] = {0, 1, 2, 3, 4, 7};
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const int q = cc[t];
      const double dqx =
          __dadd_rn(div_by(fx.f[q][k + 1], g.dx, rdx), div_by(-fx.f[q][k], g.dx, rdx));
      const double dqy =
          __dadd_rn(div_by(fy.f[q][k + g.pitch], g.dy, rdy), div_by(-fy.f[q][k], g.dy, rdy));
      const double d = __dadd_rn(-dqx, -dqy);
      out.c[q][k] = combine(un.c[q][k], b == 0.0 ? 0.0 : us.c[q][k], d);
    }
  }
  if (j < g.ny) {
    const double d = __dadd_rn(div_by(-ez[k + g.pitch], g.dy, rdy), div_by(ez[k], g.dy, rdy));
    out.c[5][k] = combine(un.c[5][k], b == 0.0 ? 0.0 : us.c[5][k], d);
  }
  if (i < g.nx) {
    const double d = __dadd_rn(div_by(ez[k + 1], g.dx, rdx), div_by(-ez[k], g.dx, rdx));
    out.c[6][k] = combine(un.c[6][k], b == 0.0 ? 0.0 : us.c[6][k], d);
  }
}

// b_update two cells at a time, every load and store of the pair one
// 16-byte double2 access (the pair's first padded column is even and the
// pitch is even, so each pair is aligned); the per-cell arithmetic and the
// cells written are b_update's.  Reads of the pair's partner beyond the
// updated range stay inside their padded rows from two ghost layers on: the
// pitch, and with it nx, is even, so they end at column nx + 1, and at row ny.
__device__ __forceinline__ double2 ld2(const double* p) {
  return __ldg(reinterpret_cast<const double2*>(p));
}
__device__ __forceinline__ void st_pair(double* p, bool a, bool b, double va, double vb) {
  if (a && b) *reinterpret_cast<double2*>(p) = make_double2(va, vb);
  else if (a) p[0] = va;
  else if (b) p[1] = vb;
}
__global__ void __launch_bounds__(256) k_update2(Grid g, StateP un, StateP us, StateP out,
                                                 FluxP fx, FluxP fy, const double* ez,
                                                 const double* dt_dev, double dt_host, int stage,
                                                 const Ctl* ctl) {
  const int pr = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int ia = 2 * pr - g.ng;  // the pair is cells ia, ia + 1 (padded columns 2 pr, 2 pr + 1)
  if (ia > g.nx || j > g.ny) return;
  if (ctl->status) return;
  const double dt = dt_dev ? *dt_dev : dt_host;
  double a, b, c;
  if (stage == 0) {
    a = 1.0; b = 0.0; c = dt;
  } else if (stage == 1) {
    a = 3.0 / 4.0; b = 1.0 / 4.0; c = (1.0 / 4.0) * dt;
  } else {
    a = 1.0 / 3.0; b = 2.0 / 3.0; c = (2.0 / 3.0) * dt;
  }
  auto combine = [&](double vn, double vs, double d) {
    if (b == 0.0) return __dadd_rn(__dmul_rn(a, vn), __dmul_rn(c, d));
    return crsum3(__dmul_rn(a, vn), __dmul_rn(b, vs), __dmul_rn(c, d));
  };
  const long long k = g.idx(ia, j), P = g.pitch;
  const double rdx = pow2_recip(g.dx), rdy = pow2_recip(g.dy);
  const int ib = ia + 1;
  // cell-centred components: i < nx, j < ny
  const bool ca = j < g.ny && ia >= 0 && ia < g.nx, cb = j < g.ny && ib >= 0 && ib < g.nx;
  if (ca || cb) {
    const int cc[6] = {0, 1, 2, 3, 4, 7};
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const int q = cc[t];
      const double2 x01 = ld2(fx.f[q] + k);
      const double x2 = __ldg(fx.f[q] + k + 2);
      const double2 y0 = ld2(fy.f[q] + k), y1 = ld2(fy.f[q] + k + P);
      const double dxa = __dadd_rn(div_by(x01.y, g.dx, rdx), div_by(-x01.x, g.dx, rdx));
      const double dxb = __dadd_rn(div_by(x2, g.dx, rdx), div_by(-x01.y, g.dx, rdx));
      const double dya = __dadd_rn(div_by(y1.x, g.dy, rdy), div_by(-y0.x, g.dy, rdy));
      const double dyb = __dadd_rn(div_by(y1.y, g.dy, rdy), div_by(-y0.y, g.dy, rdy));
      const double2 vn = ld2(un.c[q] + k);
      const double2 vs = b == 0.0 ? make_double2(0.0, 0.0) : ld2(us.c[q] + k);
      st_pair(out.c[q] + k, ca, cb, combine(vn.x, vs.x, __dadd_rn(-dxa, -dya)),
              combine(vn.y, vs.y, __dadd_rn(-dxb, -dyb)));
    }
  }
  const double2 e0 = ld2(ez + k);
  // x-face field: i <= nx, j < ny
  const bool fa = j < g.ny && ia >= 0, fb = j < g.ny && ib >= 0 && ib <= g.nx;
  if (fa || fb) {
    const double2 e1 = ld2(ez + k + P);
    const double2 vn = ld2(un.c[5] + k);
    const double2 vs = b == 0.0 ? make_double2(0.0, 0.0) : ld2(us.c[5] + k);
    const double da = __dadd_rn(div_by(-e1.x, g.dy, rdy), div_by(e0.x, g.dy, rdy));
    const double db = __dadd_rn(div_by(-e1.y, g.dy, rdy), div_by(e0.y, g.dy, rdy));
    st_pair(out.c[5] + k, fa, fb, combine(vn.x, vs.x, da), combine(vn.y, vs.y, db));
  }
  // y-face field: i < nx, j <= ny
  const bool ha = ia >= 0 && ia < g.nx, hb = ib >= 0 && ib < g.nx;
  if (ha || hb) {
    const double e2 = __ldg(ez + k + 2);
    const double2 vn = ld2(un.c[6] + k);
    const double2 vs = b == 0.0 ? make_double2(0.0, 0.0) : ld2(us.c[6] + k);
    const double da = __dadd_rn(div_by(e0.y, g.dx, rdx), div_by(-e0.x, g.dx, rdx));
    const double db = __dadd_rn(div_by(e2, g.dx, rdx), div_by(-e0.y, g.dx, rdx));
    st_pair(out.c[6] + k, ha, hb, combine(vn.x, vs.x, da), combine(vn.y, vs.y, db));
  }
}

__global__ void __launch_bounds__(256) k_update(Grid g, StateP un, StateP us, StateP out,
                                                FluxP fx, FluxP fy, const double* ez,
                                                const double* dt_dev, double dt_host, int stage,
                                                const Ctl* ctl) {
  b_update(g, un, us, out, fx, fy, ez, dt_dev, dt_host, stage, ctl, blockIdx.x, blockIdx.y);
}

// Consume the live-state preflights computed with the previous state and
// reset the per-step reductions.  coll selects which collocation the
// admissibility preflight uses (mhd_solver.cpp:689-692); anchor_mode >= 0
// forces the low-order anchor flag, -1 derives it from the live state.
__device__ __forceinline__ void k_step_begin_body(Ctl* ctl, int coll, int anchor_mode) {
  if (ctl->status) return;
  int st = 0;
  if ((coll ? ctl->anchor_theta : ctl->live_theta) != dbits(1.0)) st |= kStatusNotAdmissible;
  const double res = __longlong_as_double((long long)ctl->divb_res);
  const double sc = __longlong_as_double((long long)ctl->divb_scale);
  const double rel = res == 0.0 ? 0.0 : res / sc;
  if (!(isfinite(rel) && rel <= 1024.0 * kEps)) st |= kStatusNotSolenoidal;
  ctl->anchor_ok = anchor_mode >= 0 ? anchor_mode : (ctl->anchor_theta == dbits(1.0) ? 1 : 0);
  ctl->status = st;
  ctl->theta = dbits(1.0);
  ctl->max_rate = 0ull;
  ctl->live_theta = dbits(1.0);
  ctl->anchor_theta = dbits(1.0);
  ctl->divb_res = 0ull;
  ctl->divb_scale = 0ull;
}
__global__ void k_step_begin(Ctl* ctl, int coll, int anchor_mode) { k_step_begin_body(ctl, coll, anchor_mode); }

// Clear the status word and the live-state accumulators before the live
// state's preflights are recomputed.
__global__ void k_reset_stats(Ctl* ctl) {
  ctl->status = 0;
  ctl->live_theta = dbits(1.0);
  ctl->anchor_theta = dbits(1.0);
  ctl->divb_res = 0ull;
  ctl->divb_scale = 0ull;
}

__device__ __forceinline__ void k_set_time_body(Ctl* ctl, double t, double t_end) {
  ctl->t = t;
  ctl->t_end = t_end;
  ctl->steps_done = 0;
  ctl->status = 0;
}
__global__ void k_set_time(Ctl* ctl, double t, double t_end) { k_set_time_body(ctl, t, t_end); }

// dt = cfl_eff / max_rate (mhd_solver.cpp:1283-1320), optionally clipped to
// the remaining interval of a device-resident run.
__device__ __forceinline__ void k_dt_body(Ctl* ctl, double cfl_eff, double hmin, double hmax, int clip) {
  if (ctl->status) return;
  const double mr = __longlong_as_double((long long)ctl->max_rate);
  if (!isfinite(mr)) {
    ctl->status |= kStatusCflNonFinite;
    return;
  }
  double dt = mr > 0.0 ? cfl_eff / mr : cfl_eff * (hmin / (1.0 + hmin / hmax));
  if (clip) {
    const double rem = ctl->t_end - ctl->t;
    if (!(rem > 0.0)) {
      ctl->status |= kStatusDone;
      return;
    }
    dt = fmin(dt, rem);
  }
  ctl->dt = dt;
}
__global__ void k_dt(Ctl* ctl, double cfl_eff, double hmin, double hmax, int clip) { k_dt_body(ctl, cfl_eff, hmin, hmax, clip); }

__device__ __forceinline__ void k_step_end_body(Ctl* ctl) {
  if (ctl->status) return;
  const double rem = ctl->t_end - ctl->t;
  ctl->t = ctl->dt == rem ? ctl->t_end : ctl->t + ctl->dt;
  ctl->steps_done += 1;
  if (!(ctl->t < ctl->t_end)) ctl->status |= kStatusDone;
}
__global__ void k_step_end(Ctl* ctl) { k_step_end_body(ctl); }

__global__ void k_divb_linf(Grid g, StateP u, unsigned long long* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny || !g.in_window(i, j)) return;
  const long long k = g.idx(i, j);
  // ct_divb_linf_kernel (mhd_reduce.hip:505-553)
  const double rdx = pow2_recip(g.dx), rdy = pow2_recip(g.dy);
  const double d = __dadd_rn(__dadd_rn(div_by(u.c[5][k + 1], g.dx, rdx), div_by(-u.c[5][k], g.dx, rdx)),
                             __dadd_rn(div_by(u.c[6][k + g.pitch], g.dy, rdy),
                                       div_by(-u.c[6][k], g.dy, rdy)));
  const double v = isfinite(d) ? fabs(d) : kInf;
  atomic_max_lanes(out, v > 0.0 ? dbits(v) : 0ull);
}

// Per-block compensated partial sums of rho and energy over the cells.
__global__ void k_cell_sums(Grid g, StateP u, double* partial) {
  __shared__ double sm[2][256], sc[2][256];
  const int tid = threadIdx.x;
  double s0 = 0.0, c0 = 0.0, s1 = 0.0, c1 = 0.0;
  const long long n = (long long)g.nx * g.ny;
  for (long long t = blockIdx.x * (long long)blockDim.x + tid; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = int(t % g.nx), j = int(t / g.nx);
    if (!g.in_window(i, j)) continue;
    const long long k = g.idx(i, j);
    double e;
    two_sum(s0, u.c[0][k], s0, e);
    c0 += e;
    two_sum(s1, u.c[4][k], s1, e);
    c1 += e;
  }
  sm[0][tid] = s0; sc[0][tid] = c0;
  sm[1][tid] = s1; sc[1][tid] = c1;
  __syncthreads();
  if (tid == 0) {
    double a[2] = {0, 0}, ca[2] = {0, 0};
    for (int q = 0; q < 2; ++q)
      for (int t = 0; t < (int)blockDim.x; ++t) {
        double e;
        two_sum(a[q], sm[q][t], a[q], e);
        ca[q] += e + sc[q][t];
      }
    partial[4 * blockIdx.x + 0] = a[0];
    partial[4 * blockIdx.x + 1] = ca[0];
    partial[4 * blockIdx.x + 2] = a[1];
    partial[4 * blockIdx.x + 3] = ca[1];
  }
}

}  // namespace

// ===========================================================================
// Batched persistent kernels: each CTA walks the phase's tile list over all
// instances (stride gridDim.x), decodes (instance, tile) from the prefix
// table and runs the same device body as the single-instance kernel.
// ===========================================================================
namespace {

// (the component-wise pass, MODE 2, is memory-latency bound: 64 registers,
// eight blocks per SM; the characteristic pass needs 128)
template <int DIR, int ORDER, int MODE = 0>
__global__ void __launch_bounds__(128, MODE == 2 ? 8 : 4) kb_reconstruct(const BatchRec* __restrict__ r, BatchPlan p,
                                                      const BatchLearnRec* __restrict__ l = nullptr) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local, bx, by;
    const int inst = batch_locate(p, t, &local);
    const BatchRec& q = r[inst];
    batch_block(DIR == 0 ? kBpRecon0 : kBpRecon1, q.a.g, local, &bx, &by);
    FaceList defer{};
    if (MODE == 2)
      defer = FaceList{l[inst].flag, DIR == 0 ? l[inst].xlist : l[inst].ylist,
                       l[inst].counts + DIR};
    b_reconstruct<DIR, ORDER, MODE>(q.a.g, q.a.u, DIR == 0 ? q.a.ix : q.a.iy, q.a.gamma,
                                    q.a.ctl, bx, by, nullptr, defer);
  }
}

// Characteristic pass over every instance's face list: each CTA takes its
// share of each instance's list in turn.
template <int DIR, int ORDER>
__global__ void __launch_bounds__(128, 4) kb_reconstruct_list(const BatchRec* __restrict__ r,
                                                              const BatchLearnRec* __restrict__ l,
                                                              int n) {
  // Work units are the 32-entry chunks of every instance's list, numbered
  // across the instances in order; warp w of the grid takes chunks w, w + W,
  // ... and walks the instances' chunk counts (device values, warp-uniform)
  // alongside, so that many small lists run side by side instead of one
  // list at a time.  A chunk is the same 32 entries the single-instance
  // list pass gives a warp.
  extern __shared__ double dsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* ws = dsm + warp * kWarpReconDoubles;
  const long long stride = (long long)gridDim.x * kReconWarps;
  long long c = (long long)blockIdx.x * kReconWarps + warp;  // this warp's next chunk
  long long first = 0;  // number of the first chunk of instance `inst`
  for (int inst = 0; inst < n;) {
    const BatchRec& q = r[inst];
    const int cnt = (q.a.ctl->status & ~kStatusDone) ? 0 : l[inst].counts[DIR];
    const long long chunks = (cnt + 31) / 32;
    if (c >= first + chunks) {
      first += chunks;
      ++inst;
      continue;
    }
    const int t = int(c - first) * 32 + lane;
    const bool valid = t < cnt;
    const Grid& g = q.a.g;
    int i = 0, j = 0;
    if (valid) {
      const int k = (DIR == 0 ? l[inst].xlist : l[inst].ylist)[t];
      i = k % g.pitch - g.ng;
      j = k / g.pitch - g.ng;
    }
    mp_faces_warp<DIR, ORDER>(g, q.a.u, DIR == 0 ? q.a.ix : q.a.iy, q.a.gamma, i, j, valid, ws);
    c += stride;
  }
}

__global__ void kb_learned_reset(const BatchRec* __restrict__ r, const BatchLearnRec* __restrict__ l,
                                 BatchPlan p) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local;
    const int inst = batch_locate(p, t, &local);
    const long long k = (long long)local * 256 + threadIdx.x;
    if (k < r[inst].a.g.size()) l[inst].flag[k] = 1;
    if (local == 0 && threadIdx.x < 2) l[inst].counts[threadIdx.x] = 0;
  }
}

// k_face_lists over 256-cell chunks of every instance.
__global__ void kb_face_lists(const BatchRec* __restrict__ r, const BatchLearnRec* __restrict__ l,
                              BatchPlan p) {
  for (int tt = blockIdx.x; tt < p.total; tt += gridDim.x) {
    int local;
    const int inst = batch_locate(p, tt, &local);
    const Grid& g = r[inst].a.g;
    const BatchLearnRec& L = l[inst];
    const long long t = (long long)local * 256 + threadIdx.x;
    const unsigned lane = threadIdx.x & 31;
    bool nx_ = false, ny_ = false;
    const int k = int(t);
    if (t < g.size()) {
      const int i = int(t % g.pitch) - g.ng, j = int(t / g.pitch) - g.ng;
      if (i >= 0 && i <= g.nx && j < g.ny + g.ng) nx_ = (L.flag[t] | L.flag[t - 1]) != 0;
      if (j >= 0 && j <= g.ny && i < g.nx + g.ng) ny_ = (L.flag[t] | L.flag[t - g.pitch]) != 0;
    }
    const unsigned bx_ = __ballot_sync(0xffffffffu, nx_), by_ = __ballot_sync(0xffffffffu, ny_);
    int basex = 0, basey = 0;
    if (lane == 0) {
      if (bx_) basex = atomicAdd(&L.counts[0], __popc(bx_));
      if (by_) basey = atomicAdd(&L.counts[1], __popc(by_));
    }
    basex = __shfl_sync(0xffffffffu, basex, 0);
    basey = __shfl_sync(0xffffffffu, basey, 0);
    const unsigned below = (1u << lane) - 1u;
    if (nx_) L.xlist[basex + __popc(bx_ & below)] = k;
    if (ny_) L.ylist[basey + __popc(by_ & below)] = k;
  }
}

template <int DIR, int ORDER>
__global__ void __launch_bounds__(kFqThreads, kFqBlocksPerSm)
    kb_face_flux_q(const BatchRec* __restrict__ r, BatchPlan p, int speeds) {
  __shared__ __align__(16) double sm[ORDER == 5 ? fq_smem<DIR, 5>() : 2];
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local, bx, by;
    const BatchRec& q = r[batch_locate(p, t, &local)];
    batch_block(kBpFlux, q.a.g, local, &bx, &by);
    b_face_flux_qs<DIR, ORDER, ORDER == 7, kFqTX>(q.a.g, DIR == 0 ? q.a.ix : q.a.iy, DIR == 0 ? q.a.fx : q.a.fy,
                               DIR == 0 ? q.a.xemf : q.a.yemf, DIR == 0 ? q.a.xnj : q.a.ynj,
                               speeds ? (DIR == 0 ? q.a.xspd : q.a.yspd) : nullptr, q.a.gamma,
                               q.a.ctl, bx, by, sm);
    __syncthreads();  // the shared tile is reused by the next tile
  }
}

template <int ORDER>
__global__ void __launch_bounds__(256, 3) kb_cell_emf_s(const BatchRec* __restrict__ r, BatchPlan p,
                                                     int cfl_reduce) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local, bx, by;
    const BatchRec& q = r[batch_locate(p, t, &local)];
    batch_block(kBpCell, q.a.g, local, &bx, &by);
    b_cell_emf_s<ORDER>(q.a.g, q.a.u, q.a.cell_ez, q.a.xspd, q.a.yspd, cfl_reduce, q.a.gamma,
                        q.a.ctl, bx, by);
    __syncthreads();  // shared tiles are reused by the next tile
  }
}

template <int ORDER>
__global__ void __launch_bounds__(256, 4) kb_corner_emf_s(const BatchRec* __restrict__ r,
                                                          BatchPlan p) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local, bx, by;
    const BatchRec& q = r[batch_locate(p, t, &local)];
    batch_block(kBpCorner, q.a.g, local, &bx, &by);
    b_corner_emf_s<ORDER>(q.a.g, q.a.cell_ez, q.a.xemf, q.a.yemf, q.a.xnj, q.a.ynj, q.a.ez,
                          q.a.ctl, bx, by);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) kb_update(const BatchRec* __restrict__ r, BatchPlan p,
                                                 int stage) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local, bx, by;
    const BatchRec& q = r[batch_locate(p, t, &local)];
    batch_block(kBpUpdate, q.a.g, local, &bx, &by);
    b_update(q.a.g, q.live, q.a.u, q.out, q.a.fx, q.a.fy, q.a.ez, &q.a.ctl->dt, 0.0, stage,
             q.a.ctl, bx, by);
  }
}

__global__ void __launch_bounds__(256) kb_fill_ghosts(const BatchRec* __restrict__ r, BatchPlan p,
                                                      int axis) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local;
    const BatchRec& q = r[batch_locate(p, t, &local)];
    b_fill_ghosts(q.a.g, q.out, axis, local);
  }
}

template <int W>
__global__ void __launch_bounds__(256, 3) kb_colloc_check(const BatchRec* __restrict__ r,
                                                       BatchPlan p, int theta_mask,
                                                       int live_checks) {
  for (int t = blockIdx.x; t < p.total; t += gridDim.x) {
    int local, bx, by;
    const BatchRec& q = r[batch_locate(p, t, &local)];
    batch_block(kBpColloc, q.a.g, local, &bx, &by);
    b_colloc_check<W>(q.a.g, q.out, q.live, 1, theta_mask, live_checks, 1, q.a.gamma, q.a.ctl,
                      bx, by);
  }
}

__global__ void kb_ctl(const BatchRec* __restrict__ r, int n, int what, double t0, double t_end) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const BatchRec& q = r[k];
  Ctl* ctl = q.a.ctl;
  if (what == 0) k_step_begin_body(ctl, 0, -1);
  else if (what == 1) k_dt_body(ctl, q.cfl_eff, q.hmin, q.hmax, 1);
  else if (what == 2) k_step_end_body(ctl);
  else k_set_time_body(ctl, t0, t_end);
}

}  // namespace

// ===========================================================================
// Launch wrappers
// ===========================================================================
namespace {
inline unsigned cdiv(long long a, int b) { return unsigned((a + b - 1) / b); }

// Raise a kernel's dynamic shared-memory limit once (per process).
void ensure_smem(const void* fn, size_t bytes) {
  static std::mutex mu;
  static std::vector<const void*> done;
  std::lock_guard<std::mutex> lock(mu);
  if (std::find(done.begin(), done.end(), fn) != done.end()) return;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
  done.push_back(fn);
}
}  // namespace

void launch_fill_ghosts(const Grid& g, const StateP& u, cudaStream_t s) {
  for (int axis = 0; axis < 2; ++axis) {
    const long long n = 2LL * g.ng * ((axis == 0 ? g.ny : g.nx) + 2 * g.ng);
    k_fill_ghosts<<<cdiv(n, 256), 256, 0, s>>>(g, u, axis);
  }
}

void launch_colloc_check(const Grid& g, const StateP& cand, const StateP* base, int theta_mask,
                         bool /*anchor_check*/, bool live_checks, bool solver_owned,
                         double gamma, Ctl* ctl, cudaStream_t s) {
  const dim3 block(kBX, 8);
  const dim3 grid(cdiv(g.nx + 2 * g.ng, kBX), cdiv(g.ny + 2 * g.ng, 8));
  const StateP b = base ? *base : cand;
  const int hb = base ? 1 : 0;
  switch (g.ng) {
    case 2:
      k_colloc_check<4><<<grid, block, 0, s>>>(g, cand, b, hb, theta_mask, live_checks,
                                               solver_owned, gamma, ctl);
      break;
    case 3:
      k_colloc_check<6><<<grid, block, 0, s>>>(g, cand, b, hb, theta_mask, live_checks,
                                               solver_owned, gamma, ctl);
      break;
    default:
      k_colloc_check<8><<<grid, block, 0, s>>>(g, cand, b, hb, theta_mask, live_checks,
                                               solver_owned, gamma, ctl);
  }
}

// dir 0 or 1: that direction's faces; 2: both.
template <int ORDER>
static void recon_launch(const StageArgs& a, int dir, cudaStream_t s) {
  const Grid& g = a.g;
  const dim3 block(kBX, 4);
  const int ni = dir == 0 ? g.nx + 1 : g.nx + 2 * g.ng;
  const int nj = dir == 1 ? g.ny + 1 : g.ny + 2 * g.ng;
  const dim3 grid(cdiv(ni, kBX), cdiv(nj, 4), dir == 2 ? 2 : 1);
  size_t smem = 0;
  if (ORDER == 5 || ORDER == 7) {
    smem = kReconWarpSmem;
    ensure_smem((const void*)k_reconstruct<ORDER>, smem);
  }
  k_reconstruct<ORDER><<<grid, block, smem, s>>>(g, a.u, a.ix, a.iy, a.gamma, a.ctl,
                                                 dir == 1 ? 1 : 0);
}

void launch_reconstruct(const StageArgs& a, int dir, cudaStream_t s) {
  switch (a.order) {
    case 1: return recon_launch<1>(a, dir, s);
    case 2: return recon_launch<2>(a, dir, s);
    case 5: return recon_launch<5>(a, dir, s);
    default: return recon_launch<7>(a, dir, s);
  }
}

template <int DIR, int ORDER>
static void flux_low_launch(const StageArgs& a, bool speeds, cudaStream_t s) {
  const Grid& g = a.g;
  const dim3 block(kBX, 4);
  const dim3 grid(cdiv(g.nx + 1, kBX), cdiv(g.ny + 1, 4));
  k_face_flux<DIR, ORDER><<<grid, block, 0, s>>>(
      g, DIR == 0 ? a.ix : a.iy, DIR == 0 ? a.fx : a.fy, DIR == 0 ? a.xemf : a.yemf,
      DIR == 0 ? a.xnj : a.ynj, speeds ? (DIR == 0 ? a.xspd : a.yspd) : nullptr, a.gamma, a.ctl);
}
template <int ORDER>
static void flux_launch(const StageArgs& a, int dir, bool speeds, cudaStream_t s) {
  const Grid& g = a.g;
  const dim3 grid(cdiv(g.nx + 1, kFqTX), cdiv(g.ny + 1, fq_ty<ORDER>()), dir == 2 ? 2 : 1);
  const FaceOut ox{a.fx, a.xemf, a.xnj, speeds ? a.xspd : nullptr};
  const FaceOut oy{a.fy, a.yemf, a.ynj, speeds ? a.yspd : nullptr};
  if constexpr (ORDER == 7) {
    if ((long long)grid.x * grid.y > kFqPairBlocks) {
      const dim3 one(grid.x, grid.y);
      if (dir != 1)
        k_face_flux_one<0, ORDER><<<one, kFqThreads, 0, s>>>(g, a.ix, a.fx, a.xemf, a.xnj, ox.spd,
                                                             a.gamma, a.ctl);
      if (dir != 0)
        k_face_flux_one<1, ORDER><<<one, kFqThreads, 0, s>>>(g, a.iy, a.fy, a.yemf, a.ynj, oy.spd,
                                                             a.gamma, a.ctl);
      return;
    }
  }
  k_face_flux_qs<ORDER><<<grid, kFqThreads, 0, s>>>(g, a.ix, a.iy, ox, oy, a.gamma, a.ctl,
                                                    dir == 1 ? 1 : 0);
}

void launch_face_flux(const StageArgs& a, int dir, bool speeds, cudaStream_t s) {
  switch (a.order) {
    case 1:
      if (dir != 1) flux_low_launch<0, 1>(a, speeds, s);
      if (dir != 0) flux_low_launch<1, 1>(a, speeds, s);
      break;
    case 2:
      if (dir != 1) flux_low_launch<0, 2>(a, speeds, s);
      if (dir != 0) flux_low_launch<1, 2>(a, speeds, s);
      break;
    case 5: return flux_launch<5>(a, dir, speeds, s);
    default: return flux_launch<7>(a, dir, speeds, s);
  }
}

template <int ORDER>
static void cell_tiled_launch(const StageArgs& a, bool cfl_reduce, cudaStream_t s) {
  const Grid& g = a.g;
  const dim3 grid(cdiv(g.nx + 1, kCellTX), cdiv(g.ny + 1, kCellTY));
  if (a.cell_map) {
    constexpr size_t tbytes = sizeof(double) * cell_smem_doubles<ORDER, true>();
    ensure_smem((const void*)k_cell_emf_tma<ORDER>, tbytes);
    k_cell_emf_tma<ORDER><<<grid, dim3(kCellTX, kCellTY), tbytes, s>>>(
        g, a.u, *a.cell_map, a.cell_ez, a.xspd, a.yspd, cfl_reduce ? 1 : 0, a.gamma, a.ctl);
    return;
  }
  constexpr size_t bytes = sizeof(double) * cell_smem_doubles<ORDER>();
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(k_cell_emf_s<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(bytes));
    configured = true;
  }
  k_cell_emf_s<ORDER><<<grid, dim3(kCellTX, kCellTY), bytes, s>>>(
      g, a.u, a.cell_ez, a.xspd, a.yspd, cfl_reduce ? 1 : 0, a.gamma, a.ctl);
}

void launch_cell_emf(const StageArgs& a, bool cfl_reduce, cudaStream_t s) {
  const Grid& g = a.g;
  if (a.order == 5) return cell_tiled_launch<5>(a, cfl_reduce, s);
  if (a.order == 7) return cell_tiled_launch<7>(a, cfl_reduce, s);
  const dim3 block(kBX, 4);
  const dim3 grid(cdiv(g.nx + 1, kBX), cdiv(g.ny + 1, 4));
  const int r = cfl_reduce ? 1 : 0;
  switch (a.order) {
    case 1: k_cell_emf<1><<<grid, block, 0, s>>>(g, a.u, a.cell_ez, a.xspd, a.yspd, r, a.ctl); break;
    default: k_cell_emf<2><<<grid, block, 0, s>>>(g, a.u, a.cell_ez, a.xspd, a.yspd, r, a.ctl);
  }
}

bool make_state_tensor_map(const StateP& u, const Grid& g, int order, CUtensorMap* map) {
  if (order != 5 && order != 7) return false;
  const long long n = g.size();
  if ((g.pitch & 1) || (n & 1)) return false;  // 16-byte strides
  for (int c = 0; c < 8; ++c)
    if (u.c[c] != u.c[0] + c * n) return false;
  if (u.bxc != u.c[0] + 8 * n || u.byc != u.c[0] + 9 * n) return false;
  if (reinterpret_cast<uintptr_t>(u.c[0]) & 15) return false;
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  if (!encode) return false;
  const int sy = kCellTY + 2 * (order == 7 ? 3 : 2);
  cuuint64_t dims[3] = {cuuint64_t(g.pitch), cuuint64_t(g.ny + 2 * g.ng), 10};
  cuuint64_t strides[2] = {cuuint64_t(g.pitch) * sizeof(double), cuuint64_t(n) * sizeof(double)};
  cuuint32_t box[3] = {cuuint32_t(kTmaBW), cuuint32_t(sy), 1};
  cuuint32_t elem[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, u.c[0], dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

void launch_corner_emf(const StageArgs& a, cudaStream_t s) {
  const Grid& g = a.g;
  const dim3 tiles(cdiv(g.nx + 1, 32), cdiv(g.ny + 1, kCornerTY));
  const dim3 block(kBX, 4);
  const dim3 grid(cdiv(g.nx + 1, kBX), cdiv(g.ny + 1, 4));
  switch (a.order) {
    case 1:
    case 2: k_corner_emf<2><<<grid, block, 0, s>>>(g, a.cell_ez, a.xemf, a.yemf, a.xnj, a.ynj, a.ez, a.ctl); break;
    case 5: k_corner_emf_s<5><<<tiles, dim3(32, 8), 0, s>>>(g, a.cell_ez, a.xemf, a.yemf, a.xnj, a.ynj, a.ez, a.ctl); break;
    default: k_corner_emf_s<7><<<tiles, dim3(32, 8), 0, s>>>(g, a.cell_ez, a.xemf, a.yemf, a.xnj, a.ynj, a.ez, a.ctl);
  }
}

void launch_update(const StageArgs& a, const StateP& un, const StateP& us, const StateP& out,
                   int stage, const double* dt_dev, double dt_host, cudaStream_t s) {
  const Grid& g = a.g;
  const dim3 block(kBX, 8);
  // the paired form needs an even pitch, 16-byte aligned arrays and two ghost
  // layers (a pair's partner reads stay inside the padded arrays: at most two
  // columns past the last face, in a row before the last).  MUSCL 1024^2:
  // update 0.263 -> 0.184 ms per step.
  bool pairs = (g.pitch % 2) == 0 && g.ng >= 2;
  auto al = [](const double* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  for (int q = 0; q < 8 && pairs; ++q)
    pairs = al(un.c[q]) && al(us.c[q]) && al(out.c[q]) && al(a.fx.f[q]) && al(a.fy.f[q]);
  pairs = pairs && al(a.ez);
  if (pairs) {
    const dim3 grid(cdiv((g.nx + g.ng + 2) / 2, kBX), cdiv(g.ny + 1, 8));
    k_update2<<<grid, block, 0, s>>>(g, un, us, out, a.fx, a.fy, a.ez, dt_dev, dt_host, stage,
                                     a.ctl);
    return;
  }
  const dim3 grid(cdiv(g.nx + 1, kBX), cdiv(g.ny + 1, 8));
  k_update<<<grid, block, 0, s>>>(g, un, us, out, a.fx, a.fy, a.ez, dt_dev, dt_host, stage, a.ctl);
}

void launch_step_begin(Ctl* ctl, int coll, int anchor_mode, cudaStream_t s) {
  k_step_begin<<<1, 1, 0, s>>>(ctl, coll, anchor_mode);
}
void launch_reset_stats(Ctl* ctl, cudaStream_t s) { k_reset_stats<<<1, 1, 0, s>>>(ctl); }
void launch_set_time(Ctl* ctl, double t, double t_end, cudaStream_t s) {
  k_set_time<<<1, 1, 0, s>>>(ctl, t, t_end);
}

void launch_dt(Ctl* ctl, double cfl_eff, double hmin, double hmax, int clip, cudaStream_t s) {
  k_dt<<<1, 1, 0, s>>>(ctl, cfl_eff, hmin, hmax, clip);
}

void launch_step_end(Ctl* ctl, cudaStream_t s) { k_step_end<<<1, 1, 0, s>>>(ctl); }

void launch_divb_linf(const Grid& g, const StateP& u, unsigned long long* out, cudaStream_t s) {
  const dim3 block(kBX, 8);
  const dim3 grid(cdiv(g.nx, kBX), cdiv(g.ny, 8));
  k_divb_linf<<<grid, block, 0, s>>>(g, u, out);
}

void launch_cell_sums(const Grid& g, const StateP& u, double* partial, int blocks, cudaStream_t s) {
  k_cell_sums<<<blocks, 256, 0, s>>>(g, u, partial);
}

// ---- tile halo exchange on the device ---------------------------------------
// Gather and scatter one component by storage index.  Bad indices and
// non-finite values are recorded in *bad (bit 0: index outside [0, size),
// bit 1: non-finite value); the scatter runs as a check pass and a write
// pass, and the write pass does nothing once the check recorded a problem,
// so a rejected scatter leaves the component untouched.
__global__ void k_gather_values(const double* __restrict__ src, const long long* __restrict__ idx,
                                long long n, long long size, double* __restrict__ out,
                                unsigned long long* bad) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += stride) {
    const long long i = idx[k];
    if (i < 0 || i >= size) {
      atomicOr(bad, 1ull);
      out[k] = 0.0;
    } else {
      out[k] = src[i];
    }
  }
}

__global__ void k_scatter_check(const long long* __restrict__ idx, const double* __restrict__ v,
                                long long n, long long size, unsigned long long* bad) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long b = 0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += stride) {
    const long long i = idx[k];
    if (i < 0 || i >= size) b |= 1ull;
    if (!isfinite(v[k])) b |= 2ull;
  }
  if (b) atomicOr(bad, b);
}

__global__ void k_scatter_values(double* __restrict__ dst, const long long* __restrict__ idx,
                                 const double* __restrict__ v, long long n,
                                 const unsigned long long* bad) {
  if (*bad) return;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += stride)
    dst[idx[k]] = v[k];
}

// Any non-finite value among v[0..n) sets *bad (which must start at zero).
__global__ void k_flag_nonfinite(const double* __restrict__ v, long long n,
                                 unsigned long long* bad) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  bool b = false;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += stride)
    b = b || !isfinite(v[k]);
  if (__any_sync(0xffffffffu, b) && (threadIdx.x & 31) == 0) atomicOr(bad, 1ull);
}

namespace {
int exchange_blocks(long long n) {
  const long long b = (n + 255) / 256;
  return (int)(b < 4 * 148 ? (b > 0 ? b : 1) : 4 * 148);
}
}  // namespace

// y[k] = rcp_nr(x[k]), z[k] = rsqrt_nr(x[k]) (the accuracy test's hook).
__global__ void k_probe_roots(const double* __restrict__ x, long long n, double* y, double* z) {
  const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  y[k] = rcp_nr(x[k]);
  z[k] = rsqrt_nr(x[k]);
}
__global__ void k_probe_quotients(const double* __restrict__ a, const double* __restrict__ b,
                                  long long n, double* q) {
  const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  SharedDiv d;
  const double v = d.by(b[k]).of(a[k]);
  q[k] = d.bad ? __ddiv_rn(a[k], b[k]) : v;
}
// The reconstruction's eigen-system of the states u[0..8)[n] (x-normal): whether
// its bound skips the L R = I check, and max |L R - I| of the rows and columns it
// would project with.
__global__ void k_probe_eigen(const double* __restrict__ u, long long n, double gamma, int* sure,
                              double* err) {
  const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const Eg e = eig_scalars(St{u[k], u[n + k], u[2 * n + k], u[3 * n + k], u[4 * n + k], u[5 * n + k],
                              u[6 * n + k], u[7 * n + k]}, gamma);
  sure[k] = e.sure;
  double L[7][7], R[7][7];
  for (int r = 0; r < 4; ++r) {
    WavePair w;
    wave_pair(e, r, w);
    for (int m = 0; m < 7; ++m) {
      const double lv = m < 4 && r < 3 ? w.lv[m] : 0.0;
      const double rv = m > 0 && m < 5 && r < 3 ? w.rv[m - 1] : 0.0;
      L[r][m] = w.lt[m] - lv;
      R[r][m] = w.rt[m] - rv;
      L[6 - r][m] = w.lt[m] + lv;
      R[6 - r][m] = w.rt[m] + rv;
    }
  }
  double worst = 0.0;
  for (int a = 0; a < 7; ++a)
    for (int b = 0; b < 7; ++b) {
      double s = a == b ? -1.0 : 0.0;
      for (int m = 0; m < 7; ++m) s = fma(L[a][m], R[b][m], s);
      worst = fabs(s) <= worst ? worst : fabs(s);  // NaN stays
    }
  err[k] = worst;
}
void launch_probe_eigen(const double* u, long long n, double gamma, int* sure, double* err,
                        cudaStream_t s) {
  if (n > 0) k_probe_eigen<<<cdiv(n, 128), 128, 0, s>>>(u, n, gamma, sure, err);
}
void launch_probe_quotients(const double* a, const double* b, long long n, double* q,
                            cudaStream_t s) {
  if (n > 0) k_probe_quotients<<<cdiv(n, 256), 256, 0, s>>>(a, b, n, q);
}
void launch_probe_roots(const double* x, long long n, double* y, double* z, cudaStream_t s) {
  if (n > 0) k_probe_roots<<<cdiv(n, 256), 256, 0, s>>>(x, n, y, z);
}

void launch_flag_nonfinite(const double* v, long long n, unsigned long long* bad, cudaStream_t s) {
  if (n <= 0) return;
  k_flag_nonfinite<<<exchange_blocks(n), 256, 0, s>>>(v, n, bad);
}

void launch_gather_values(const double* src, const long long* idx, long long n, long long size,
                          double* out, unsigned long long* bad, cudaStream_t s) {
  if (n <= 0) return;
  k_gather_values<<<exchange_blocks(n), 256, 0, s>>>(src, idx, n, size, out, bad);
}

void launch_scatter_values(double* dst, const long long* idx, const double* v, long long n,
                           long long size, unsigned long long* bad, cudaStream_t s) {
  if (n <= 0) return;
  k_scatter_check<<<exchange_blocks(n), 256, 0, s>>>(idx, v, n, size, bad);
  k_scatter_values<<<exchange_blocks(n), 256, 0, s>>>(dst, idx, v, n, bad);
}

// ---- batched launchers -----------------------------------------------------
namespace {
template <class K>
int max_ctas(K kernel, int threads, size_t smem) {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) != cudaSuccess) b = 1;
  return b > 0 ? b : 1;
}
inline unsigned pgrid(const BatchPlan& p) { return unsigned(p.grid > 0 ? p.grid : p.total); }

template <int ORDER>
void batch_cell_configure() {
  static bool done = false;
  if (!done) {
    cudaFuncSetAttribute(kb_cell_emf_s<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(sizeof(double) * cell_smem_doubles<ORDER>()));
    done = true;
  }
}
}  // namespace

int batch_phase_threads(int phase) {
  switch (phase) {
    case kBpRecon0: case kBpRecon1: return 128;
    case kBpFlux: return kFqThreads;
    default: return 256;
  }
}

int batch_phase_max_ctas_per_sm(int phase, int order) {
  const bool o7 = order == 7;
  switch (phase) {
    case kBpRecon0:
      ensure_smem((const void*)kb_reconstruct<0, 7>, kReconWarpSmem);
      ensure_smem((const void*)kb_reconstruct<0, 5>, kReconWarpSmem);
      return o7 ? max_ctas(kb_reconstruct<0, 7>, 128, kReconWarpSmem)
                : max_ctas(kb_reconstruct<0, 5>, 128, kReconWarpSmem);
    case kBpRecon1:
      ensure_smem((const void*)kb_reconstruct<1, 7>, kReconWarpSmem);
      ensure_smem((const void*)kb_reconstruct<1, 5>, kReconWarpSmem);
      return o7 ? max_ctas(kb_reconstruct<1, 7>, 128, kReconWarpSmem)
                : max_ctas(kb_reconstruct<1, 5>, 128, kReconWarpSmem);
    case kBpFlux: {
      constexpr int t = kFqThreads;
      return o7 ? max_ctas(kb_face_flux_q<0, 7>, t, 0) : max_ctas(kb_face_flux_q<0, 5>, t, 0);
    }
    case kBpCell:
      if (o7) {
        batch_cell_configure<7>();
        return max_ctas(kb_cell_emf_s<7>, 256, sizeof(double) * cell_smem_doubles<7>());
      }
      batch_cell_configure<5>();
      return max_ctas(kb_cell_emf_s<5>, 256, sizeof(double) * cell_smem_doubles<5>());
    case kBpCorner: return o7 ? max_ctas(kb_corner_emf_s<7>, 256, 0) : max_ctas(kb_corner_emf_s<5>, 256, 0);
    case kBpUpdate: return max_ctas(kb_update, 256, 0);
    case kBpColloc: return o7 ? max_ctas(kb_colloc_check<8>, 256, 0) : max_ctas(kb_colloc_check<6>, 256, 0);
    default: return max_ctas(kb_fill_ghosts, 256, 0);
  }
}

void launch_batch_reconstruct(const BatchRec* r, const BatchPlan& p, int dir, int order,
                              cudaStream_t s) {
  const dim3 block(32, 4);
  if (order == 7) {
    if (dir == 0) {
      ensure_smem((const void*)kb_reconstruct<0, 7>, kReconWarpSmem);
      kb_reconstruct<0, 7><<<pgrid(p), block, kReconWarpSmem, s>>>(r, p);
    } else {
      ensure_smem((const void*)kb_reconstruct<1, 7>, kReconWarpSmem);
      kb_reconstruct<1, 7><<<pgrid(p), block, kReconWarpSmem, s>>>(r, p);
    }
  } else {
    if (dir == 0) {
      ensure_smem((const void*)kb_reconstruct<0, 5>, kReconWarpSmem);
      kb_reconstruct<0, 5><<<pgrid(p), block, kReconWarpSmem, s>>>(r, p);
    } else {
      ensure_smem((const void*)kb_reconstruct<1, 5>, kReconWarpSmem);
      kb_reconstruct<1, 5><<<pgrid(p), block, kReconWarpSmem, s>>>(r, p);
    }
  }
}

void launch_batch_face_flux(const BatchRec* r, const BatchPlan& p, int dir, int order,
                            bool speeds, cudaStream_t s) {
  const int sp = speeds ? 1 : 0;
  if (order == 7) {
    if (dir == 0) kb_face_flux_q<0, 7><<<pgrid(p), kFqThreads, 0, s>>>(r, p, sp);
    else kb_face_flux_q<1, 7><<<pgrid(p), kFqThreads, 0, s>>>(r, p, sp);
  } else {
    if (dir == 0) kb_face_flux_q<0, 5><<<pgrid(p), kFqThreads, 0, s>>>(r, p, sp);
    else kb_face_flux_q<1, 5><<<pgrid(p), kFqThreads, 0, s>>>(r, p, sp);
  }
}

void launch_batch_cell_emf(const BatchRec* r, const BatchPlan& p, int order, bool cfl_reduce,
                           cudaStream_t s) {
  const dim3 block(kCellTX, kCellTY);
  if (order == 7) {
    batch_cell_configure<7>();
    kb_cell_emf_s<7><<<pgrid(p), block, sizeof(double) * cell_smem_doubles<7>(), s>>>(
        r, p, cfl_reduce ? 1 : 0);
  } else {
    batch_cell_configure<5>();
    kb_cell_emf_s<5><<<pgrid(p), block, sizeof(double) * cell_smem_doubles<5>(), s>>>(
        r, p, cfl_reduce ? 1 : 0);
  }
}

void launch_batch_corner_emf(const BatchRec* r, const BatchPlan& p, int order, cudaStream_t s) {
  const dim3 block(32, 8);
  if (order == 7) kb_corner_emf_s<7><<<pgrid(p), block, 0, s>>>(r, p);
  else kb_corner_emf_s<5><<<pgrid(p), block, 0, s>>>(r, p);
}

void launch_batch_update(const BatchRec* r, const BatchPlan& p, int stage, cudaStream_t s) {
  kb_update<<<pgrid(p), dim3(32, 8), 0, s>>>(r, p, stage);
}

void launch_batch_fill_ghosts(const BatchRec* r, const BatchPlan& p, int axis, cudaStream_t s) {
  kb_fill_ghosts<<<pgrid(p), 256, 0, s>>>(r, p, axis);
}

void launch_batch_colloc_check(const BatchRec* r, const BatchPlan& p, int order, int theta_mask,
                               bool live_checks, cudaStream_t s) {
  const dim3 block(32, 8);
  if (order == 7) kb_colloc_check<8><<<pgrid(p), block, 0, s>>>(r, p, theta_mask, live_checks ? 1 : 0);
  else kb_colloc_check<6><<<pgrid(p), block, 0, s>>>(r, p, theta_mask, live_checks ? 1 : 0);
}

void launch_batch_learned_reset(const BatchRec* r, const BatchLearnRec* l, const BatchPlan& cells,
                                cudaStream_t s) {
  kb_learned_reset<<<pgrid(cells), 256, 0, s>>>(r, l, cells);
}

void launch_batch_face_lists(const BatchRec* r, const BatchLearnRec* l, const BatchPlan& cells,
                             cudaStream_t s) {
  kb_face_lists<<<pgrid(cells), 256, 0, s>>>(r, l, cells);
}

void launch_batch_reconstruct_learned(const BatchRec* r, const BatchLearnRec* l,
                                      const BatchPlan& p, int dir, int order, int list_grid,
                                      cudaStream_t s) {
  const dim3 block(32, 4);
  if (order == 7) {
    if (dir == 0) {
      kb_reconstruct<0, 7, 2><<<pgrid(p), block, 0, s>>>(r, p, l);
      ensure_smem((const void*)kb_reconstruct_list<0, 7>, kReconWarpSmem);
      kb_reconstruct_list<0, 7><<<list_grid, 128, kReconWarpSmem, s>>>(r, l, p.n);
    } else {
      kb_reconstruct<1, 7, 2><<<pgrid(p), block, 0, s>>>(r, p, l);
      ensure_smem((const void*)kb_reconstruct_list<1, 7>, kReconWarpSmem);
      kb_reconstruct_list<1, 7><<<list_grid, 128, kReconWarpSmem, s>>>(r, l, p.n);
    }
  } else {
    if (dir == 0) {
      kb_reconstruct<0, 5, 2><<<pgrid(p), block, 0, s>>>(r, p, l);
      ensure_smem((const void*)kb_reconstruct_list<0, 5>, kReconWarpSmem);
      kb_reconstruct_list<0, 5><<<list_grid, 128, kReconWarpSmem, s>>>(r, l, p.n);
    } else {
      kb_reconstruct<1, 5, 2><<<pgrid(p), block, 0, s>>>(r, p, l);
      ensure_smem((const void*)kb_reconstruct_list<1, 5>, kReconWarpSmem);
      kb_reconstruct_list<1, 5><<<list_grid, 128, kReconWarpSmem, s>>>(r, l, p.n);
    }
  }
}

void launch_batch_ctl(const BatchRec* r, int n, int what, double t, double t_end, cudaStream_t s) {
  kb_ctl<<<cdiv(n, 128), 128, 0, s>>>(r, n, what, t, t_end);
}

// ---- learned-mode reconstruction and indicator training data ----------------
namespace {
template <int DIR, int ORDER>
dim3 recon_grid(const Grid& g) {
  const int ni = DIR == 0 ? g.nx + 1 : g.nx + 2 * g.ng;
  const int nj = DIR == 0 ? g.ny + 2 * g.ng : g.ny + 1;
  return dim3(cdiv(ni, kBX), cdiv(nj, 4));
}
}  // namespace

void launch_reconstruct_label(const StageArgs& a, int dir, int* label, int literal,
                              cudaStream_t s) {
  const dim3 block(kBX, 4);
  const IfaceP out = dir == 0 ? a.ix : a.iy;
#define QB_LBL(D, O)                                                                          \
  if (dir == D && a.order == O) {                                                            \
    ensure_smem((const void*)k_reconstruct_label<D, O>, kReconSmem);                          \
    return (void)k_reconstruct_label<D, O><<<recon_grid<D, O>(a.g), block, kReconSmem, s>>>( \
        a.g, a.u, out, a.gamma, a.ctl, label, literal);                                       \
  }
  QB_LBL(0, 5) QB_LBL(1, 5) QB_LBL(0, 7) QB_LBL(1, 7)
#undef QB_LBL
}

void launch_reconstruct_learned(const StageArgs& a, int dir, const unsigned char* flag, int* list,
                                int* count, int list_grid, cudaStream_t s) {
  const dim3 block(kBX, 4);
  const IfaceP out = dir == 0 ? a.ix : a.iy;
  const FaceList defer{flag, list, count};
#define QB_LRN(D, O)                                                                            \
  if (dir == D && a.order == O) {                                                              \
    k_reconstruct_lin<D, O><<<recon_grid<D, O>(a.g), block, 0, s>>>(a.g, a.u, out, a.gamma,    \
                                                                    a.ctl, defer);             \
    ensure_smem((const void*)k_reconstruct_list<D, O>, kReconWarpSmem);                         \
    k_reconstruct_list<D, O><<<list_grid, 128, kReconWarpSmem, s>>>(a.g, a.u, out, a.gamma, a.ctl,   \
                                                                list, count);                  \
    return;                                                                                    \
  }
  QB_LRN(0, 5) QB_LRN(1, 5) QB_LRN(0, 7) QB_LRN(1, 7)
#undef QB_LRN
}

void launch_face_lists(const Grid& g, const unsigned char* flag, int* xlist, int* ylist,
                       int* counts, cudaStream_t s) {
  cudaMemsetAsync(counts, 0, 2 * sizeof(int), s);
  k_face_lists<<<cdiv(g.size(), 256), 256, 0, s>>>(g, flag, xlist, ylist, counts);
}

// ===========================================================================
// Kernels of the per-kernel launch interface (reference
// include/quasar/physics/mhd/kernels.hpp): the pieces that the fused step
// above combines (flux difference, EMF curl, stage combine) as separate
// launches, plus standalone forms of the reductions and fills.  Each uses the
// arithmetic of the fused kernel it stands beside, so a step composed from
// these launches reproduces the fused step.
// ===========================================================================
namespace {

// Never written: the status word every stage kernel polls reads 0.
__device__ Ctl g_abi_zero_ctl;

// dudt += -(F_hi - F_lo)/h over the interior cells, all eight slots
// (mhd_update.hip:21-105).
__global__ void __launch_bounds__(256) k_abi_flux_difference(Grid g, FluxP f, int dir, FluxP d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const long long k = g.idx(i, j), kp = k + (dir == 0 ? 1 : g.pitch);
  const double h = dir == 0 ? g.dx : g.dy, rh = pow2_recip(h);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const double dq = __dadd_rn(div_by(f.f[q][kp], h, rh), div_by(-f.f[q][k], h, rh));
    d.f[q][k] = __dadd_rn(d.f[q][k], -dq);
  }
}

// dudt.bx_face / dudt.by_face = curl of the corner E_z, overwritten
// (mhd_ct.hip:893-931): bx on i <= nx, j < ny; by on i < nx, j <= ny.
__global__ void __launch_bounds__(256) k_abi_curl_rate(Grid g, const double* __restrict__ ez,
                                                       double* dbx, double* dby) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i > g.nx || j > g.ny) return;
  const long long k = g.idx(i, j);
  const double rdx = pow2_recip(g.dx), rdy = pow2_recip(g.dy);
  if (j < g.ny) dbx[k] = __dadd_rn(div_by(-ez[k + g.pitch], g.dy, rdy), div_by(ez[k], g.dy, rdy));
  if (i < g.nx) dby[k] = __dadd_rn(div_by(ez[k + 1], g.dx, rdx), div_by(-ez[k], g.dx, rdx));
}

// out = a un + b us + c dudt (mhd_update.hip:113-206): an operand whose weight
// is zero is not read, (1, 0, 0) is an exact copy; cell components over the
// interior, bx also on i = nx and by on j = ny.
__global__ void __launch_bounds__(256) k_abi_rk_stage(Grid g, StateP out, StateP un, StateP us,
                                                      FluxP d, double a, double b, double c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i > g.nx || j > g.ny) return;
  const long long k = g.idx(i, j);
  const bool copy = a == 1.0 && b == 0.0 && c == 0.0;
  const bool ua = a != 0.0, ub = b != 0.0, uc = c != 0.0;
  auto comb = [&](int q) {
    if (copy) return un.c[q][k];
    if (ua && ub && uc)
      return crsum3(__dmul_rn(a, un.c[q][k]), __dmul_rn(b, us.c[q][k]), __dmul_rn(c, d.f[q][k]));
    if (ua && ub) return __dadd_rn(__dmul_rn(a, un.c[q][k]), __dmul_rn(b, us.c[q][k]));
    if (ua && uc) return __dadd_rn(__dmul_rn(a, un.c[q][k]), __dmul_rn(c, d.f[q][k]));
    if (ub && uc) return __dadd_rn(__dmul_rn(b, us.c[q][k]), __dmul_rn(c, d.f[q][k]));
    if (ua) return __dmul_rn(a, un.c[q][k]);
    if (ub) return __dmul_rn(b, us.c[q][k]);
    if (uc) return __dmul_rn(c, d.f[q][k]);
    return 0.0;
  };
  if (i < g.nx && j < g.ny) {
    const int cc[6] = {0, 1, 2, 3, 4, 7};
#pragma unroll
    for (int t = 0; t < 6; ++t) out.c[cc[t]][k] = comb(cc[t]);
  }
  if (j < g.ny) out.c[5][k] = comb(5);
  if (i < g.nx) out.c[6][k] = comb(6);
}

// Face -> cell collocation of one axis over the padded grid
// (launch_mhd_collocate_face_to_cell, mhd_staggering.hpp:77-236).
template <int W>
__global__ void k_abi_collocate(Grid g, int axis, const double* __restrict__ face,
                                double* __restrict__ cell) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x - g.ng;
  const int j = blockIdx.y * blockDim.y + threadIdx.y - g.ng;
  if (i >= g.nx + g.ng || j >= g.ny + g.ng) return;
  cell[g.idx(i, j)] = axis == 0
                          ? face_to_cell<W>(face, (long long)g.idx(0, j), 1, i, -g.ng, g.nx + g.ng - 1)
                          : face_to_cell<W>(face, (long long)g.idx(i, 0), g.pitch, j, -g.ng,
                                            g.ny + g.ng - 1);
}

// ---- analytic initial state (mhd_initial_conditions.hip:59-340) -----------
// Status bits of kernels.hpp:650-655.
constexpr int kSeedDensity = 1, kSeedPressure = 2, kSeedMomentum = 4, kSeedEnergy = 8,
              kSeedCollocation = 16, kSeedCoordinate = 32;

struct SeedW {
  double rho, p, vx, vy, vz, bx, by, bz, eoff;
};

// The generators in the reference's operation order, every product and sum
// rounded on its own (no contraction); sin, cos and hypot are CUDA's.
__device__ SeedW seed_eval(const SeedSpec& s, int nx, double xc, double yc) {
  constexpr double kPi = 3.141592653589793;  // nearest double to pi
  const double two_pi = 2.0 * kPi;
  SeedW w{};
  switch (s.kind) {
    case 0: {  // brio_wu: left/right primitive states split at x = interface
      const double* side = xc < s.interface_x ? s.left : s.right;
      w.rho = side[0]; w.p = side[1]; w.vx = side[2]; w.vy = side[3]; w.vz = side[4];
      w.bx = side[5]; w.by = side[6]; w.bz = side[7];
      break;
    }
    case 1: {  // alfven_wave along x with the sinc cell-average factor
      const double n = double(s.wavenumber);
      const double k = __ddiv_rn(__dmul_rn(two_pi, n), s.lx);
      const double phase = __dmul_rn(k, __dsub_rn(xc, s.ox));
      const double q = __ddiv_rn(n, double(nx));
      double fv = 1.0;
      if (q != 0.0) {
        const double pq = __dmul_rn(kPi, q);
        fv = __ddiv_rn(sin(pq), pq);
      }
      const double inv = __ddiv_rn(copysign(s.mvs, s.total_b0), __dsqrt_rn(s.rho));
      const double sp = sin(phase), cp = cos(phase);
      const double a = __dmul_rn(__dmul_rn(-s.amplitude, inv), fv);
      w.rho = s.rho; w.p = s.pressure; w.vx = 0.0;
      w.vy = __dmul_rn(a, sp);
      w.vz = __dmul_rn(a, cp);
      w.bx = s.b0;
      w.by = __dmul_rn(__dmul_rn(s.amplitude, fv), sp);
      w.bz = __dmul_rn(__dmul_rn(s.amplitude, fv), cp);
      const double sa = __dmul_rn(s.amplitude, s.mvs);
      w.eoff = __dmul_rn(__dmul_rn(sa, sa), __dsub_rn(1.0, __dmul_rn(fv, fv)));
      break;
    }
    case 2: {  // orszag_tang
      const double xi = __ddiv_rn(__dsub_rn(xc, s.ox), s.lx);
      const double eta = __ddiv_rn(__dsub_rn(yc, s.oy), s.ly);
      const double b0 = s.b_uniform[0];
      const double se = sin(__dmul_rn(two_pi, eta));
      w.rho = __dmul_rn(s.gamma, s.gamma); w.p = s.gamma;
      w.vx = -se;
      w.vy = sin(__dmul_rn(two_pi, xi));
      w.bx = __dmul_rn(-b0, se);
      w.by = __dmul_rn(b0, sin(__dmul_rn(2.0 * two_pi, xi)));
      break;
    }
    case 3: {  // blast: pressure disk
      const double r = hypot(__dsub_rn(xc, s.center[0]), __dsub_rn(yc, s.center[1]));
      w.rho = s.rho_ambient;
      w.p = r < s.r_in ? s.p_core : s.p_ambient;
      w.bx = s.b_uniform[0]; w.by = s.b_uniform[1]; w.bz = s.b_uniform[2];
      break;
    }
    case 4: {  // rotor: rigid disk with a linear taper
      const double rx = __dsub_rn(xc, s.center[0]), ry = __dsub_rn(yc, s.center[1]);
      const double r = hypot(rx, ry);
      double f = __ddiv_rn(__dsub_rn(s.r1, r), __dsub_rn(s.r1, s.r0));
      f = fmin(fmax(f, 0.0), 1.0);
      const bool inside = r <= s.r0;
      if (inside) f = 1.0;
      if (r >= s.r1) f = 0.0;
      double speed = 0.0;
      if (inside) speed = __ddiv_rn(s.u0, s.r0);
      else if (r < s.r1) speed = __ddiv_rn(__dmul_rn(f, s.u0), r);
      w.rho = __dadd_rn(s.rho_out, __dmul_rn(f, __dsub_rn(s.rho_in, s.rho_out)));
      w.p = s.p_ambient;
      w.vx = __dmul_rn(-speed, ry);
      w.vy = __dmul_rn(speed, rx);
      w.bx = s.b_uniform[0]; w.by = s.b_uniform[1]; w.bz = s.b_uniform[2];
      break;
    }
    default: {  // confined_blob: dense square, uniform bz
      const bool inside = fabs(__dsub_rn(xc, s.center[0])) <= s.blob_half &&
                          fabs(__dsub_rn(yc, s.center[1])) <= s.blob_half;
      w.rho = inside ? s.rho_in : s.rho_out;
      w.p = inside ? s.p_in : s.p_out;
      w.bz = s.b_uniform[2];
      break;
    }
  }
  return w;
}

// Pass 1 (mhd_initial_conditions.hip:211-282): one padded cell per thread;
// the faces of a cell take its centre value.
__global__ void __launch_bounds__(256) k_seed_pass1(Grid g, SeedSpec s, StateP u, double* raw,
                                                    int* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x - g.ng;
  const int j = blockIdx.y * blockDim.y + threadIdx.y - g.ng;
  if (i >= g.nx + g.ng || j >= g.ny + g.ng) return;
  const double xc = fma(double(i) + 0.5, g.dx, s.ox);
  const double yc = fma(double(j) + 0.5, g.dy, s.oy);
  if (!(isfinite(xc) && isfinite(yc))) {
    atomicOr(status, kSeedCoordinate);
    return;
  }
  const SeedW w = seed_eval(s, g.nx, xc, yc);
  if (!(isfinite(w.rho) && w.rho > 0.0)) {
    atomicOr(status, kSeedDensity);
    return;
  }
  if (!(isfinite(w.p) && w.p > 0.0)) {
    atomicOr(status, kSeedPressure);
    return;
  }
  const double kinetic = kin_vel(w.rho, w.vx, w.vy, w.vz);
  const double magnetic = half_sq3(w.bx, w.by, w.bz);
  const double energy = __dadd_rn(
      __dadd_rn(__dadd_rn(__ddiv_rn(w.p, __dsub_rn(s.gamma, 1.0)), kinetic), magnetic), w.eoff);
  const double mx = __dmul_rn(w.rho, w.vx), my = __dmul_rn(w.rho, w.vy),
               mz = __dmul_rn(w.rho, w.vz);
  if (!(isfinite(mx) && isfinite(my) && isfinite(mz))) {
    atomicOr(status, kSeedMomentum);
    return;
  }
  if (!isfinite(energy)) {
    atomicOr(status, kSeedEnergy);
    return;
  }
  const long long k = g.idx(i, j);
  u.c[0][k] = w.rho;
  u.c[1][k] = mx;
  u.c[2][k] = my;
  u.c[3][k] = mz;
  u.c[4][k] = energy;
  u.c[5][k] = __dmul_rn(s.magnetic_scale, w.bx);
  u.c[6][k] = __dmul_rn(s.magnetic_scale, w.by);
  u.c[7][k] = __dmul_rn(s.magnetic_scale, w.bz);
  raw[k] = magnetic;
}

// Pass 2 (mhd_initial_conditions.hip:284-340): E = (E - raw) + |B_c|^2 / 2
// with B_c the collocated field the solver's EOS reads, then the preflight
// on the conserved arrays.
__global__ void __launch_bounds__(256) k_seed_recollocate(Grid g, double gamma, StateP u,
                                                          const double* raw, int* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x - g.ng;
  const int j = blockIdx.y * blockDim.y + threadIdx.y - g.ng;
  if (i >= g.nx + g.ng || j >= g.ny + g.ng) return;
  const long long k = g.idx(i, j);
  const double bxc = u.bxc[k], byc = u.byc[k];
  if (!(isfinite(bxc) && isfinite(byc))) {
    atomicOr(status, kSeedCollocation);
    return;
  }
  const double adjusted =
      __dadd_rn(__dsub_rn(u.c[4][k], raw[k]), half_sq3(bxc, byc, u.c[7][k]));
  if (!isfinite(adjusted)) {
    atomicOr(status, kSeedEnergy);
    return;
  }
  u.c[4][k] = adjusted;
  const double rho = u.c[0][k];
  if (!(isfinite(rho) && rho > 0.0)) {
    atomicOr(status, kSeedDensity);
    return;
  }
  const St st{rho, u.c[1][k], u.c[2][k], u.c[3][k], adjusted, bxc, byc, u.c[7][k]};
  const double p = pressure(st, gamma);
  if (!isfinite(p)) {
    atomicOr(status, kSeedEnergy);
    return;
  }
  if (!(p > 0.0)) atomicOr(status, kSeedPressure);
}

// One side's ghost layers, fluid (parts 1) or field (parts 2)
// (mhd_boundary_hip.hip:66-218).
__global__ void k_abi_fill_side(Grid g, StateP u, int side, int mode, int parts) {
  const int axis = side / 2;
  const int lines = (axis == 0 ? g.ny : g.nx) + 2 * g.ng;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.ng * lines) return;
  fill_ghost(g, u, axis, (side & 1) == 0, mode, t / lines + 1, t % lines - g.ng, parts);
}

__device__ __forceinline__ void atomic_min_lanes(unsigned long long* dst, unsigned long long v) {
  const cg::coalesced_group grp = cg::coalesced_threads();
  const unsigned long long m = cg::reduce(grp, v, cg::less<unsigned long long>());
  if (grp.thread_rank() == 0) atomicMin(dst, m);
}

// Cell state with the high-order (coll 0) or two-face (coll 1) collocated
// in-plane field, formed from the face arrays (mhd_staggering.hpp:321-338).
template <int W>
__device__ __forceinline__ St abi_cell(const Grid& g, const StateP& u, int i, int j, int coll) {
  if (coll) return load_cell1(u, g, i, j);
  const long long k = g.idx(i, j);
  return St{u.c[0][k], u.c[1][k], u.c[2][k], u.c[3][k], u.c[4][k],
            face_to_cell<W>(u.c[5], (long long)g.idx(0, j), 1, i, -g.ng, g.nx + g.ng - 1),
            face_to_cell<W>(u.c[6], (long long)g.idx(i, 0), g.pitch, j, -g.ng, g.ny + g.ng - 1),
            u.c[7][k]};
}

// Admissible convex fraction with density and internal-energy floors
// (mhd_reduce.hip:143-209); *theta holds the bits of the running minimum.
template <int W>
__global__ void __launch_bounds__(256) k_abi_admissible(Grid g, StateP base, StateP cand,
                                                        double rho_floor, double q_floor,
                                                        int coll, unsigned long long* theta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const St a = abi_cell<W>(g, base, i, j, coll), b = abi_cell<W>(g, cand, i, j, coll);
  double local = 1.0;
  const double qa = convex_q(a, b, 0.0);
  if (!(a.rho > rho_floor) || !(qa > q_floor) || !isfinite(a.rho) || !isfinite(qa)) {
    local = 0.0;
  } else if (!(isfinite(b.rho) && isfinite(b.mx) && isfinite(b.my) && isfinite(b.mz) &&
               isfinite(b.E) && isfinite(b.bx) && isfinite(b.by) && isfinite(b.bz))) {
    local = 0.0;
  } else {
    double hi = 1.0;
    if (b.rho <= rho_floor) {
      const double den = a.rho - b.rho;
      hi = den > 0.0 ? (a.rho - rho_floor) / den : 0.0;
      hi = fmin(fmax(hi, 0.0), 1.0);
    }
    if (convex_q(a, b, hi) > q_floor) {
      local = hi;
    } else {
      double lo = 0.0;
      for (int it = 0; it < 56; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (convex_q(a, b, mid) > q_floor) lo = mid;
        else hi = mid;
      }
      local = lo;
    }
  }
  atomic_min_lanes(theta, dbits(local));
}

// Relative solenoidality of the interior cells: acc[0] residual, acc[1]
// scale maxima (bits).
__global__ void __launch_bounds__(256) k_abi_divb_relative(Grid g, StateP u, int solver_owned,
                                                           unsigned long long* acc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  unsigned long long rb, sb;
  divb_cell(g, u, g.idx(i, j), solver_owned, rb, sb);
  atomic_max_lanes(acc, rb);
  atomic_max_lanes(acc + 1, sb);
}

// CFL rate 0.5 alpha / h of the face with high cell (i, j) normal to DIR, as
// the face-flux kernels form it: the face-average Riemann problem and, for
// MP5/MP7, every Gauss point before the first inadmissible one
// (mhd_reduce.hip:254-416).
template <int DIR, int ORDER>
__device__ double abi_face_rate(const Grid& g, const IfaceP& in, int i, int j, double gamma) {
  int si = i, sj = j;
  if (DIR == 0 && i == g.nx && g.bc[0] == 0 && g.bc[1] == 0) si = 0;
  if (DIR == 1 && j == g.ny && g.bc[2] == 0 && g.bc[3] == 0) sj = 0;
  const long long ks = g.idx(si, sj);
  const double h = DIR == 0 ? g.dx : g.dy;
  const St bl = iface(in, ks, true), br = iface(in, ks, false);
  double rate = face_rate<DIR, ORDER>(bl, br, gamma, h, rcp_rho(bl.rho), rcp_rho(br.rho));
  if (ORDER != 5 && ORDER != 7) return rate;
  constexpr int H = ORDER == 5 ? 2 : 3, N = 2 * H + 1, Q = ORDER == 5 ? 3 : 4;
  const long long ts = DIR == 0 ? g.pitch : 1;
  for (int q = 0; q < Q; ++q) {
    double pl[8], pr[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      double sa[N], sb[N];
#pragma unroll
      for (int t = 0; t < N; ++t) {
        sa[t] = in.L[c][ks + (t - H) * ts];
        sb[t] = in.R[c][ks + (t - H) * ts];
      }
      // the face flux's own sums: all nodes at once at MP7, one at MP5
      if (ORDER == 7) {
        double va[Q], vb[Q];
        point_values<ORDER>(sa, va);
        point_values<ORDER>(sb, vb);
        pl[c] = q == 0 ? va[0] : q == 1 ? va[1] : q == 2 ? va[2] : va[Q - 1];
        pr[c] = q == 0 ? vb[0] : q == 1 ? vb[1] : q == 2 ? vb[2] : vb[Q - 1];
      } else {
        pl[c] = point_value<ORDER>(q, sa);
        pr[c] = point_value<ORDER>(q, sb);
      }
    }
    const St l{pl[0], pl[1], pl[2], pl[3], pl[4], pl[5], pl[6], pl[7]};
    const St r{pr[0], pr[1], pr[2], pr[3], pr[4], pr[5], pr[6], pr[7]};
    if (!point_admissible(l, gamma) || !point_admissible(r, gamma)) break;
    rate = fmax(rate, face_rate<DIR, ORDER>(l, r, gamma, h, rcp_nr(l.rho), rcp_nr(r.rho)));
  }
  return rate;
}

template <int ORDER>
__global__ void __launch_bounds__(256) k_abi_cfl_rate(Grid g, IfaceP ix, IfaceP iy, double gamma,
                                                      unsigned long long* max_rate) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const double r = (abi_face_rate<0, ORDER>(g, ix, i, j, gamma) +
                    abi_face_rate<0, ORDER>(g, ix, i + 1, j, gamma)) +
                   (abi_face_rate<1, ORDER>(g, iy, i, j, gamma) +
                    abi_face_rate<1, ORDER>(g, iy, i, j + 1, gamma));
  const double local = isfinite(r) ? fmax(0.0, r) : kInf;
  atomic_max_lanes(max_rate, dbits(local));
}

__global__ void k_abi_set_u64(unsigned long long* p, int n, unsigned long long v) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) p[t] = v;
}

std::mutex g_abi_mu;
Ctl* g_abi_ctl_ptr[64] = {};

}  // namespace

cudaError_t abi_zero_ctl(Ctl** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_abi_mu);
  if (!g_abi_ctl_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_abi_zero_ctl);
    if (e != cudaSuccess) return e;
    g_abi_ctl_ptr[dev] = static_cast<Ctl*>(p);
  }
  *out = g_abi_ctl_ptr[dev];
  return cudaSuccess;
}

void launch_abi_flux_difference(const Grid& g, const FluxP& f, int dir, const FluxP& d,
                                cudaStream_t s) {
  k_abi_flux_difference<<<dim3(cdiv(g.nx, kBX), cdiv(g.ny, 8)), dim3(kBX, 8), 0, s>>>(g, f, dir, d);
}

void launch_abi_curl_rate(const Grid& g, const double* ez, double* dbx, double* dby,
                          cudaStream_t s) {
  k_abi_curl_rate<<<dim3(cdiv(g.nx + 1, kBX), cdiv(g.ny + 1, 8)), dim3(kBX, 8), 0, s>>>(g, ez, dbx,
                                                                                       dby);
}

void launch_abi_rk_stage(const Grid& g, const StateP& out, const StateP& un, const StateP& us,
                         const FluxP& d, double a, double b, double c, cudaStream_t s) {
  k_abi_rk_stage<<<dim3(cdiv(g.nx + 1, kBX), cdiv(g.ny + 1, 8)), dim3(kBX, 8), 0, s>>>(
      g, out, un, us, d, a, b, c);
}

void launch_abi_collocate(const Grid& g, int axis, const double* face, double* cell,
                          cudaStream_t s) {
  const dim3 grid(cdiv(g.nx + 2 * g.ng, kBX), cdiv(g.ny + 2 * g.ng, 8)), block(kBX, 8);
  if (g.ng == 2) k_abi_collocate<4><<<grid, block, 0, s>>>(g, axis, face, cell);
  else if (g.ng == 3) k_abi_collocate<6><<<grid, block, 0, s>>>(g, axis, face, cell);
  else k_abi_collocate<8><<<grid, block, 0, s>>>(g, axis, face, cell);
}

void launch_abi_seed(const Grid& g, const SeedSpec& spec, const StateP& out, double* raw,
                     int* status, cudaStream_t s) {
  const dim3 block(kBX, 8), grid(cdiv(g.nx + 2 * g.ng, kBX), cdiv(g.ny + 2 * g.ng, 8));
  k_seed_pass1<<<grid, block, 0, s>>>(g, spec, out, raw, status);
  launch_abi_collocate(g, 0, out.c[5], out.bxc, s);
  launch_abi_collocate(g, 1, out.c[6], out.byc, s);
  k_seed_recollocate<<<grid, block, 0, s>>>(g, spec.gamma, out, raw, status);
}

void launch_abi_fill_side(const Grid& g, const StateP& u, int side, int mode, int parts,
                          cudaStream_t s) {
  const long long n = (long long)g.ng * ((side / 2 == 0 ? g.ny : g.nx) + 2 * g.ng);
  k_abi_fill_side<<<cdiv(n, 256), 256, 0, s>>>(g, u, side, mode, parts);
}

void launch_abi_admissible(const Grid& g, const StateP& base, const StateP& cand,
                           double rho_floor, double q_floor, int coll, unsigned long long* theta,
                           cudaStream_t s) {
  const dim3 grid(cdiv(g.nx, kBX), cdiv(g.ny, 8)), block(kBX, 8);
  if (g.ng == 2) k_abi_admissible<4><<<grid, block, 0, s>>>(g, base, cand, rho_floor, q_floor, coll, theta);
  else if (g.ng == 3) k_abi_admissible<6><<<grid, block, 0, s>>>(g, base, cand, rho_floor, q_floor, coll, theta);
  else k_abi_admissible<8><<<grid, block, 0, s>>>(g, base, cand, rho_floor, q_floor, coll, theta);
}

void launch_abi_divb_relative(const Grid& g, const StateP& u, int solver_owned,
                              unsigned long long* acc, cudaStream_t s) {
  k_abi_divb_relative<<<dim3(cdiv(g.nx, kBX), cdiv(g.ny, 8)), dim3(kBX, 8), 0, s>>>(
      g, u, solver_owned, acc);
}

void launch_abi_cfl_rate(const Grid& g, const IfaceP& ix, const IfaceP& iy, int order,
                         double gamma, unsigned long long* max_rate, cudaStream_t s) {
  const dim3 grid(cdiv(g.nx, kBX), cdiv(g.ny, 8)), block(kBX, 8);
  switch (order) {
    case 1: k_abi_cfl_rate<1><<<grid, block, 0, s>>>(g, ix, iy, gamma, max_rate); break;
    case 2: k_abi_cfl_rate<2><<<grid, block, 0, s>>>(g, ix, iy, gamma, max_rate); break;
    case 5: k_abi_cfl_rate<5><<<grid, block, 0, s>>>(g, ix, iy, gamma, max_rate); break;
    default: k_abi_cfl_rate<7><<<grid, block, 0, s>>>(g, ix, iy, gamma, max_rate);
  }
}

void launch_abi_set_u64(unsigned long long* p, int n, unsigned long long v, cudaStream_t s) {
  k_abi_set_u64<<<cdiv(n, 256), 256, 0, s>>>(p, n, v);
}

}  // namespace qb
