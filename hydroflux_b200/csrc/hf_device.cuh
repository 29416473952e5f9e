// hf_device.cuh -- per-face and per-cell device arithmetic of the explicit step.
//
// Every function keeps the operation order of the Rust reference
// (franciscoparrao/hydroflux, solver-2d) so that, compiled with
// --fmad=false and IEEE division / square root, it rounds like the
// reference's f64 code. Citations are file:line in that crate.
//
// The state arithmetic is generic over the scalar T (hf_scalar.cuh): double
// for the production step, DualD for the forward-mode tangent, like the
// reference's `T: Real` code. Bed elevations are never differentiated and
// stay double; branches read values only.
#pragma once

#include <cstdint>

#include "hf_arith.h"
#include "hf_internal.h"
#include "hf_pow.h"
#include "hf_scalar.cuh"

namespace hf {

// solver-2d/src/lib.rs:43, 63, 72; riemann.rs:74; boundary.rs:68, 76
constexpr double GRAVITY = 9.81;
constexpr double H_DRY = 1.0e-6;
constexpr double H_VEL = 1.0e-5;
constexpr double DRY_TOL = 1.0e-12;
constexpr double DRY_INFLOW_SLOPE_THRESHOLD = 5.0e-4;
constexpr double DRY_INFLOW_H_MAX = 10.0;

enum { BC_TRANSMISSIVE = 0, BC_WALL = 1, BC_DISCHARGE = 2, BC_DEPTH = 3 };
enum { SIDE_NORTH = 0, SIDE_SOUTH = 1, SIDE_WEST = 2, SIDE_EAST = 3 };

template <class T> struct GhostT {
  T h, hu, hv;
  double z;
};
using Ghost = GhostT<double>;

// ghost_cell (boundary.rs:193-219) with ghost_state (274-333) and ghost_bed
// (335-367). `c0` is the boundary cell, `c1` the next cell inward along the
// face normal (only read for Discharge / Depth, which need two cells). The
// Manning value (and, for DualD, its tangent `dnman`) is read only by the
// dry-inflow Discharge ghost.
template <class T>
__device__ __forceinline__ GhostT<T> ghost_cell(int side, const BcDev& bc, T h, T hu, T hv,
                                                const double* __restrict__ z,
                                                const double* __restrict__ nman,
                                                const double* __restrict__ dnman, int64_t c0,
                                                int64_t c1, double d_normal) {
  const int kind = bc.kind[side];
  const double bval = bc.val[side];
  const bool xf = side >= SIDE_WEST;
  GhostT<T> g{h, hu, hv, 0.0};
  if (kind == BC_WALL) {
    if (xf) g.hu = -hu; else g.hv = -hv;
  } else if (kind == BC_DISCHARGE) {
    if (xf) g.hu = cst<T>(bval); else g.hv = cst<T>(bval);
  } else if (kind == BC_DEPTH) {
    g.h = cst<T>(bval);
  }
  if (kind == BC_TRANSMISSIVE || kind == BC_WALL) {
    g.z = z[c0];
  } else {
    g.z = z[c0] * 2.0 - z[c1];
  }
  if (kind == BC_DISCHARGE && val(h) < H_DRY) {
    // |bed_slope| along the normal (boundary.rs:241-271); |a-b| is exact in
    // either order, so the side-specific operand order does not matter.
    const double slope_mag = fabs(hfa::div_rn(z[c0] - z[c1], d_normal));
    if (slope_mag > DRY_INFLOW_SLOPE_THRESHOLD) {
      const T n0 = Field<T>::ld(nman, dnman, c0);
      const T h_n = r_pow35(n0 * hfa::div_rn(fabs(bval), sqrt(slope_mag)));
      g.h = r_min(h_n, cst<T>(DRY_INFLOW_H_MAX));
    }
  }
  return g;
}

// hllc_normal_flux (riemann.rs:114-204). Only the side that the sampling
// picks has its tangential velocity and star depth evaluated; those are the
// only values the reference's result reads, so the result is identical.
template <class T>
__device__ __forceinline__ void hllc_normal(T h_l, T qn_l, T qt_l, T h_r, T qn_r, T qt_r,
                                            T& o_m, T& o_n, T& o_t) {
  const bool wl = val(h_l) > DRY_TOL;
  const bool wr = val(h_r) > DRY_TOL;
  const T Z = cst<T>(0.0);
  if (!wl && !wr) {
    o_m = Z; o_n = Z; o_t = Z;
    return;
  }
  const T cl = wl ? r_sqrt_pos(h_l * GRAVITY) : Z;
  const T cr = wr ? r_sqrt_pos(h_r * GRAVITY) : Z;
  const T un_l = wl ? dvp(qn_l, h_l) : Z;  // h > DRY_TOL > 0
  const T un_r = wr ? dvp(qn_r, h_r) : Z;
  T sl, sr;
  if (wl && wr) {
    sl = r_min(un_l - cl, un_r - cr);
    sr = r_max(un_l + cl, un_r + cr);
  } else if (!wl) {
    sl = un_r - cr * 2.0;
    sr = un_r + cr;
  } else {
    sl = un_l - cl;
    sr = un_l + cl * 2.0;
  }
  bool left, star;
  T s_star = Z;
  if (val(sl) >= 0.0) {
    left = true; star = false;
  } else if (val(sr) <= 0.0) {
    left = false; star = false;
  } else {
    const T denom = h_r * (un_r - sr) - h_l * (un_l - sl);
    s_star = fabs(val(denom)) > 1.0e-12
                 ? dv(h_r * (un_r - sr) * sl - h_l * (un_l - sl) * sr, denom)
                 : (sl + sr) * 0.5;
    left = val(s_star) >= 0.0;
    star = true;
  }
  const T h = left ? h_l : h_r;
  const T qn = left ? qn_l : qn_r;
  const T qt = left ? qt_l : qt_r;
  const T un = left ? un_l : un_r;
  const bool wet = left ? wl : wr;
  const T ut = wet ? dvp(qt, h) : Z;
  T fm = Z, fn = Z, ft = Z;
  if (wet) {
    fm = qn;
    fn = qn * un + h * h * (0.5 * GRAVITY);
    ft = qn * ut;
  }
  if (!star) {
    o_m = fm; o_n = fn; o_t = ft;
    return;
  }
  const T s = left ? sl : sr;
  const T hs = dv(h * (s - un), s - s_star);
  o_m = fm + (hs - h) * s;
  o_n = fn + (hs * s_star - qn) * s;
  o_t = ft + (hs * ut - qt) * s;
}

// well_balanced_x_face / _y_face (update.rs:256-353) with z_left = z_right =
// zf (every call site passes the shared face bed). States are oriented:
// (h, normal momentum, tangential momentum). Outputs: mass, the normal
// momentum flux seen by the minus (left/top) and plus (right/bottom) cell,
// and the tangential momentum flux.
template <class T>
__device__ __forceinline__ void wb_face(T hL, T qnL, T qtL, T hR, T qnR, T qtR, double zf,
                                        T& mass, T& n_minus, T& n_plus, T& tang) {
  const double z_max = fmax(zf, zf);
  const T Z = cst<T>(0.0);
  const T hsL = r_max(hL + zf - z_max, Z);
  const T hsR = r_max(hR + zf - z_max, Z);
  T unL = Z, utL = Z, unR = Z, utR = Z;
  if (val(hL) > H_VEL) dvp2(qnL, qtL, hL, unL, utL);  // hL > H_VEL
  if (val(hR) > H_VEL) dvp2(qnR, qtR, hR, unR, utR);
  T fm, fn, ft;
  hllc_normal<T>(hsL, hsL * unL, hsL * utL, hsR, hsR * unR, hsR * utR, fm, fn, ft);
  const T corrL = (hL * hL - hsL * hsL) * (0.5 * GRAVITY);
  const T corrR = (hR * hR - hsR * hsR) * (0.5 * GRAVITY);
  mass = fm;
  n_minus = fn + corrL;
  n_plus = fn + corrR;
  tang = ft;
}

// The general face out of line, for the few faces of a moderate tile that
// wb_face_wet leaves (kept out of the loop so that its registers do not
// weigh on the common path).
struct FaceFlux {
  double mass, n_minus, n_plus, tang;
};
static __device__ __noinline__ FaceFlux wb_face_general(double hL, double qnL, double qtL, double hR,
                                                 double qnR, double qtR, double zf) {
  FaceFlux f;
  wb_face<double>(hL, qnL, qtL, hR, qnR, qtR, zf, f.mass, f.n_minus, f.n_plus, f.tang);
  return f;
}

// wb_face with both sides wet, for the faces of a tile whose inputs are all
// moderate (hfa::moderate_or_zero; depths not negative). Same operations in
// the same order, so the same values, with
// - every quotient and root by the unguarded helpers (recip_rn, quo_*,
//   sqrt_rn_moderate): six reciprocals serve the nine quotients;
// - the sides' cases dropped: h > H_VEL on both sides makes the velocities
//   plain quotients and every max(., 0) its argument, and hs > DRY_TOL makes
//   both sides wet for HLLC, whose sampling is then three selects.
// The divisors of the star state have known signs: denom < 0 (both products
// subtract a speed from a bound on it), and s - s_star < 0 on the left and
// > 0 on the right, where the numerator is >= +0, so quo_plus gives the IEEE
// zeros. Returns false, with no flux, where a condition fails or a divisor's
// low word is all ones; the caller then takes wb_face_general.
// - Comparisons read the operands' high words (the integer pipe; a compare on
//   the FP64 pipe takes twice an issue slot). Thresholds are compared strictly
//   on the high word: a value within 2^-20 above one counts as a failed
//   condition. sl and sr, sums with a root > 0, are never -0 or below 2^-253;
//   s_star may be -0, the one value with the high word 0x80000000, which is
//   >= 0. (256^2 dam break, intervals of 0.4 s: 579 -> 552 us.)
//
// Per face this is about 150 FP64 operations, two cycles of a scheduler per
// warp each. They are not the bound by themselves: on the 2048^2 valley the FP64
// pipe is 36% busy and the issue slots 57%, with barriers and dependent
// operations in the rest (profiles/stage_kernel32_valley2048.md).
__device__ __forceinline__ constexpr int high_word(double x) {  // of a positive constant
  return (int)(__builtin_bit_cast(unsigned long long, x) >> 32);
}
__device__ __forceinline__ bool wb_face_wet_q(double hL, double qnL_, double qtL_, double hR,
                                            double qnR_, double qtR_, double zf, FaceFlux& f) {
  const double hsL = hL + zf - zf, hsR = hR + zf - zf;
  const int hv = high_word(H_VEL), ht = high_word(DRY_TOL);
  if (!(__double2hiint(hL) > hv && __double2hiint(hR) > hv && __double2hiint(hsL) > ht &&
        __double2hiint(hsR) > ht))
    return false;
  bool ones = hfa::low_word_ones(hL) || hfa::low_word_ones(hR) || hfa::low_word_ones(hsL) ||
              hfa::low_word_ones(hsR);
  double y = hfa::recip_rn(hL);
  const double qnL = hsL * hfa::quo_keep(qnL_, hL, y);
  const double qtL = hsL * hfa::quo_keep(qtL_, hL, y);
  y = hfa::recip_rn(hR);
  const double qnR = hsR * hfa::quo_keep(qnR_, hR, y);
  const double qtR = hsR * hfa::quo_keep(qtR_, hR, y);
  const double yL = hfa::recip_rn(hsL), yR = hfa::recip_rn(hsR);
  const double unL = hfa::quo_keep(qnL, hsL, yL), unR = hfa::quo_keep(qnR, hsR, yR);
  const double cl = hfa::sqrt_rn_moderate(hsL * GRAVITY);
  const double cr = hfa::sqrt_rn_moderate(hsR * GRAVITY);
  const double al = unL - cl, ar = unR - cr, bl = unL + cl, br = unR + cr;
  const double sl = al < ar ? al : ar;
  const double sr = bl > br ? bl : br;
  const double tR = hsR * (unR - sr), tL = hsL * (unL - sl);
  const double denom = tR - tL;
  const double s_star = hfa::quo_plus(tR * sl - tL * sr, denom, hfa::recip_rn(denom));
  const bool slow = __double2hiint(sl) < 0;  // sl < 0
  const bool star = slow && __double2hiint(sr) > 0;
  const bool left = star ? (unsigned)__double2hiint(s_star) <= 0x80000000u : !slow;
  const double h = left ? hsL : hsR, qn = left ? qnL : qnR, qt = left ? qtL : qtR;
  const double un = left ? unL : unR, s = left ? sl : sr;
  const double ut = hfa::quo_keep(qt, h, left ? yL : yR);
  f.mass = qn;
  double fn = qn * un + h * h * (0.5 * GRAVITY);
  f.tang = qn * ut;
  if (star) {
    const double b = s - s_star;
    ones = ones || hfa::low_word_ones(denom) || hfa::low_word_ones(b) ||
           (__double2hiint(denom) & 0x7fffffff) <= high_word(1.0e-12);
    const double hs = hfa::quo_plus(h * (s - un), b, hfa::recip_rn(b));
    f.mass = qn + (hs - h) * s;
    fn = fn + (hs * s_star - qn) * s;
    f.tang = f.tang + (hs * ut - qt) * s;
  }
  f.n_minus = fn + (hL * hL - hsL * hsL) * (0.5 * GRAVITY);
  f.n_plus = fn + (hR * hR - hsR * hsR) * (0.5 * GRAVITY);
  return !ones;
}

// The same from velocities, as the reconstruction gives them.
__device__ __forceinline__ bool wb_face_wet(double hL, double unL, double utL, double hR,
                                            double unR, double utR, double zf, FaceFlux& f) {
  return wb_face_wet_q(hL, hL * unL, hL * utL, hR, hR * unR, hR * utR, zf, f);
}

// A face of a moderate tile that wb_face_wet leaves, from the reconstructed
// depths before the max(., 0): one side dry behind a step of the bed (most of
// them), or a side too thin for a velocity. The cases of wb_face and
// hllc_normal in their order, with the unguarded quotients and roots. denom is
// negative whatever side is dry (a dry side's product is a zero), and b has
// the sign it has in wb_face_wet, so the zeros of quo_plus are the IEEE ones;
// a dry side's velocities are +0. Only significands of ones are left to
// wb_face_general, about twice the work: on a flooding ensemble 17% of the
// faces, and 42% of the warps' passes over faces, come here (16 valleys of
// sides 64 to 640, 72 steps: 47.7 -> 45.1 ms; a 1-step call at 700 x 500
// 178.7 -> 171.7 us).
// Takes momenta; a negative depth's are not read.
static __device__ __noinline__ FaceFlux wb_face_moderate_q(double hm, double qn_m, double qt_m,
                                                           double hp, double qn_p, double qt_p,
                                                           double zf) {
  FaceFlux f{0.0, 0.0, 0.0, 0.0};
  const double hL = __double2hiint(hm) < 0 ? 0.0 : hm, hR = __double2hiint(hp) < 0 ? 0.0 : hp;
  if (hL == 0.0 && hR == 0.0) return f;
  double hsL = hL + zf - zf, hsR = hR + zf - zf;
  hsL = __double2hiint(hsL) < 0 ? 0.0 : hsL;
  hsR = __double2hiint(hsR) < 0 ? 0.0 : hsR;
  const bool wl = hsL > DRY_TOL, wr = hsR > DRY_TOL;
  bool ones = hfa::low_word_ones(hL) || hfa::low_word_ones(hR) || hfa::low_word_ones(hsL) ||
              hfa::low_word_ones(hsR);
  double fn = 0.0;
  if (wl || wr) {
    double qnL = 0.0, qtL = 0.0, unL = 0.0, utL = 0.0, cl = 0.0;
    double qnR = 0.0, qtR = 0.0, unR = 0.0, utR = 0.0, cr = 0.0;
    if (hL > H_VEL) {
      const double y = hfa::recip_rn(hL);
      qnL = hsL * hfa::quo_keep(qn_m, hL, y);
      qtL = hsL * hfa::quo_keep(qt_m, hL, y);
    }
    if (hR > H_VEL) {
      const double y = hfa::recip_rn(hR);
      qnR = hsR * hfa::quo_keep(qn_p, hR, y);
      qtR = hsR * hfa::quo_keep(qt_p, hR, y);
    }
    if (wl) {
      const double y = hfa::recip_rn(hsL);
      unL = hfa::quo_keep(qnL, hsL, y);
      utL = hfa::quo_keep(qtL, hsL, y);
      cl = hfa::sqrt_rn_moderate(hsL * GRAVITY);
    }
    if (wr) {
      const double y = hfa::recip_rn(hsR);
      unR = hfa::quo_keep(qnR, hsR, y);
      utR = hfa::quo_keep(qtR, hsR, y);
      cr = hfa::sqrt_rn_moderate(hsR * GRAVITY);
    }
    double sl, sr;
    if (wl && wr) {
      const double al = unL - cl, ar = unR - cr, bl = unL + cl, br = unR + cr;
      sl = al < ar ? al : ar;
      sr = bl > br ? bl : br;
    } else if (wr) {
      sl = unR - cr * 2.0;
      sr = unR + cr;
    } else {
      sl = unL - cl;
      sr = unL + cl * 2.0;
    }
    const bool star = sl < 0.0 && sr > 0.0;
    bool left = sl >= 0.0;
    double s_star = 0.0;
    if (star) {
      const double tR = hsR * (unR - sr), tL = hsL * (unL - sl);
      const double denom = tR - tL;
      ones = ones || hfa::low_word_ones(denom);
      s_star = fabs(denom) > 1.0e-12
                   ? hfa::quo_plus(tR * sl - tL * sr, denom, hfa::recip_rn(denom))
                   : (sl + sr) * 0.5;
      left = s_star >= 0.0;
    }
    const bool wet = left ? wl : wr;
    const double h = left ? hsL : hsR, qn = left ? qnL : qnR, qt = left ? qtL : qtR;
    const double un = left ? unL : unR, ut = left ? utL : utR, s = left ? sl : sr;
    if (wet) {
      f.mass = qn;
      fn = qn * un + h * h * (0.5 * GRAVITY);
      f.tang = qn * ut;
    }
    if (star) {
      const double b = s - s_star;
      ones = ones || hfa::low_word_ones(b);
      const double hs = hfa::quo_plus(h * (s - un), b, hfa::recip_rn(b));
      f.mass = f.mass + (hs - h) * s;
      fn = fn + (hs * s_star - qn) * s;
      f.tang = f.tang + (hs * ut - qt) * s;
    }
  }
  if (ones) return wb_face_general(hL, qn_m, qt_m, hR, qn_p, qt_p, zf);
  f.n_minus = fn + (hL * hL - hsL * hsL) * (0.5 * GRAVITY);
  f.n_plus = fn + (hR * hR - hsR * hsR) * (0.5 * GRAVITY);
  return f;
}

__device__ __forceinline__ FaceFlux wb_face_moderate(double hm, double un_m, double ut_m,
                                                     double hp, double un_p, double ut_p,
                                                     double zf) {
  return wb_face_moderate_q(hm, hm * un_m, hm * ut_m, hp, hp * un_p, hp * ut_p, zf);
}

// The reference's minmod(dl / d, dr / d) evaluated literally (update.rs:362-370).
template <class T> __device__ __noinline__ T minmod_literal(T dl, T dr, double d) {
  const T a = dvp(dl, d), b = dvp(dr, d);  // d = dx or dy > 0
  if (val(a) * val(b) <= 0.0) return cst<T>(0.0);
  return fabs(val(a)) < fabs(val(b)) ? a : b;
}

// minmod(dl / d, dr / d) with one division. Division by d > 0 keeps the sign
// and the weak order of the numerators, so the operand selected here has the
// quotient the reference returns (when the quotients tie, both are the same
// value). A zero difference makes the reference's product of quotients +-0,
// hence 0. Tiny or infinite operands, where the reference's product of
// quotients could underflow or be NaN, take the literal path out of line.
template <class T> __device__ __forceinline__ T minmod_div(T dl, T dr, const hfa::RecipD& rd) {
  const double l = val(dl), r = val(dr);
  const bool finite = hfa::is_finite(l) && hfa::is_finite(r);
  if ((hfa::is_zero(l) || hfa::is_zero(r)) && finite) return cst<T>(0.0);
  if (!finite || fabs(l) < 1.0e-140 || fabs(r) < 1.0e-140) return minmod_literal<T>(dl, dr, rd.d);
  if (l * r <= 0.0) return cst<T>(0.0);
  return dvr(fabs(l) < fabs(r) ? dl : dr, rd);
}

// minmod_div for moderate operands and spacing (no quotient or product of
// quotients under- or overflows): zero where the signs differ or an operand
// is zero, else the quotient of the smaller magnitude. quo_plus makes every
// zero +0, which is what the reference returns there.
__device__ __forceinline__ double minmod_moderate(double l, double r, const hfa::RecipD& rd) {
  double pick = fabs(l) < fabs(r) ? l : r;
  if ((__double2hiint(l) ^ __double2hiint(r)) < 0) pick = 0.0;
  return hfa::quo_plus(pick, rd.d, rd.hi);
}

// The stage's operations with a guarded and a moderate (MOD, f64) form.
// Limited slope of the middle one of three values.
template <class T, bool MOD>
__device__ __forceinline__ T limited_slope(T l, T c, T r, const hfa::RecipD& rd) {
  if constexpr (MOD) return minmod_moderate(c - l, r - c, rd);
  else return minmod_div<T>(c - l, r - c, rd);
}
// Unlimited slope of a cell on a side from its one difference.
template <class T, bool MOD>
__device__ __forceinline__ T side_slope(T d, const hfa::RecipD& rd) {
  if constexpr (MOD) return cst<T>(hfa::quo_keep(val(d), rd.d, rd.hi));
  else return dvr(d, rd);
}
// Face between two cells from their reconstructed depths (before the
// max(., 0)) and velocities (update.rs:560-623).
template <class T>
__device__ __forceinline__ void face_interior(T hm, T un_m, T ut_m, T hp, T un_p, T ut_p, double zf,
                                              T& m, T& n_minus, T& n_plus, T& tang) {
  const T Z = cst<T>(0.0);
  const T h_m = r_max(hm, Z), h_p = r_max(hp, Z);
  wb_face<T>(h_m, h_m * un_m, h_m * ut_m, h_p, h_p * un_p, h_p * ut_p, zf, m, n_minus, n_plus,
             tang);
}

// Which operand minmod_div(dl, dr, d) returns: -1 for the constant zero, 0
// for dl / d, 1 for dr / d. Same branches as minmod_div / minmod_literal.
__device__ __forceinline__ int minmod_pick(double l, double r, double d) {
  const bool finite = hfa::is_finite(l) && hfa::is_finite(r);
  if ((hfa::is_zero(l) || hfa::is_zero(r)) && finite) return -1;
  if (!finite || fabs(l) < 1.0e-140 || fabs(r) < 1.0e-140) {
    const double a = hfa::div_rn(l, d), b = hfa::div_rn(r, d);
    if (a * b <= 0.0) return -1;
    return fabs(a) < fabs(b) ? 0 : 1;
  }
  if (l * r <= 0.0) return -1;
  return fabs(l) < fabs(r) ? 0 : 1;
}

// Manning friction on one cell (source.rs:150-164); h^(4/3) correctly rounded.
template <class T>
__device__ __forceinline__ void friction_cell(T h, T& hu, T& hv, T n, double dt, double dry_tol) {
  if (val(h) <= dry_tol) return;
  if (val(n) == 0.0) return;
  const double dt_g = dt * GRAVITY;
  const T speed = dv(r_sqrt(hu * hu + hv * hv), h);
  const T factor = dv(n * n * speed, r_pow43(h)) * dt_g + 1.0;
  hu = dv(hu, factor);
  hv = dv(hv, factor);
}

// The same on f64 with the moderate helpers where the operands allow it:
// h, n and dt within 2^+-60 and |q|^2 within 2^+-240 keep every
// intermediate within 2^+-580 (the smaller momentum component is zero or at
// least 2^-200). Water at rest (|q|^2 = 0) keeps its momentum: its factor is
// 0 + 1.
__device__ __forceinline__ void friction_moderate(double h, double& hu, double& hv, double n,
                                                  double dt, double dry_tol) {
  if (h <= dry_tol || n == 0.0) return;
  const double dt_g = dt * GRAVITY;
  const double q2 = hu * hu + hv * hv;
  if (hfa::positive_within<60>(h) && hfa::positive_within<60>(n) &&
      hfa::positive_within<60>(dt_g)) {
    if (q2 == 0.0) return;
    if (hfa::positive_within<240>(q2) && hfa::moderate_or_zero(hu) && hfa::moderate_or_zero(hv)) {
      const double p = hfpow::pow_4_3(h);
      const double speed = hfa::quo_keep(hfa::sqrt_rn_moderate(q2), h, hfa::recip_rn(h));
      const double factor = hfa::quo_keep(n * n * speed, p, hfa::recip_rn(p)) * dt_g + 1.0;
      if (!(hfa::low_word_ones(h) || hfa::low_word_ones(p) || hfa::low_word_ones(factor))) {
        const double y = hfa::recip_rn(factor);
        hu = hfa::quo_keep(hu, factor, y);
        hv = hfa::quo_keep(hv, factor, y);
        return;
      }
    }
  }
  friction_cell<double>(h, hu, hv, n, dt, dry_tol);
}

// Piecewise-linear series (same definition as the host forcing descriptor).
__device__ __forceinline__ double series_eval(const double* ts, const double* vs, int n, double t) {
  if (n <= 0) return 0.0;
  if (n == 1 || t <= ts[0]) return vs[0];
  if (t >= ts[n - 1]) return vs[n - 1];
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (ts[mid] <= t) lo = mid; else hi = mid;
  }
  const double w = hfa::div_rn(t - ts[lo], ts[lo + 1] - ts[lo]);
  return vs[lo] + (vs[lo + 1] - vs[lo]) * w;
}

// A series with units: sampled at t / t_div, value (v * v_mul) / v_div, the
// arithmetic of a caller that keeps its hydrograph in minutes and mm/h
// (solver-2d/examples/uk_ea_test8a_official.rs:119-134). The default units
// (1, 1, 1) give series_eval exactly.
__device__ __forceinline__ double series_eval_u(const double* ts, const double* vs, int n,
                                                double t, const SeriesUnits& u) {
  const double v = series_eval(ts, vs, n, hfa::div_rn(t, u.t_div));
  return hfa::div_rn(v * u.v_mul, u.v_div);
}

// Wave speeds of an interior cell for the CFL bound (update.rs:121-135).
__device__ __forceinline__ void cell_speeds(double h, double hu, double hv, double& sx,
                                            double& sy) {
  if (h <= H_DRY) return;
  if (hfa::positive_within<60>(h) && !hfa::low_word_ones(h) && hfa::moderate_or_zero(hu) &&
      hfa::moderate_or_zero(hv)) {
    const double c = hfa::sqrt_rn_moderate(GRAVITY * h);
    double u = 0.0, v = 0.0;
    if (h > H_VEL) {
      const double y = hfa::recip_rn(h);
      u = hfa::quo_keep(hu, h, y);
      v = hfa::quo_keep(hv, h, y);
    }
    const double ax = fabs(u) + c, ay = fabs(v) + c;
    sx = ax > sx ? ax : sx;
    sy = ay > sy ? ay : sy;
    return;
  }
  {
    // NaN depth: the reference's `h <= H_DRY` is false and sqrt(NaN) is
    // folded into f64::max, which ignores NaN; fmax does the same.
    const double c = sqrt(GRAVITY * h);
    double u = 0.0, v = 0.0;
    if (h > H_VEL) {
      u = hfa::div_rn(hu, h);
      v = hfa::div_rn(hv, h);
    }
    sx = fmax(sx, fabs(u) + c);
    sy = fmax(sy, fabs(v) + c);
  }
}

// Ghost-cell wave speeds (update.rs:177-188): no H_VEL cutoff there.
__device__ __forceinline__ void ghost_speeds(const Ghost& g, double& sx, double& sy) {
  const double h = g.h;
  if (h <= H_DRY) return;
  const double c = sqrt(GRAVITY * h);
  const double u = hfa::div_rn(g.hu, h);
  const double v = hfa::div_rn(g.hv, h);
  sx = fmax(sx, fabs(u) + c);
  sy = fmax(sy, fabs(v) + c);
}

// The same for moderate ghosts; false, with nothing added, for others.
__device__ __forceinline__ bool ghost_speeds_moderate(double h, double hu, double hv, double& sx,
                                                      double& sy) {
  if (h <= H_DRY) return true;
  if (!(hfa::positive_within<60>(h) && !hfa::low_word_ones(h) && hfa::moderate_or_zero(hu) &&
        hfa::moderate_or_zero(hv)))
    return false;
  const double c = hfa::sqrt_rn_moderate(GRAVITY * h), y = hfa::recip_rn(h);
  const double ax = fabs(hfa::quo_keep(hu, h, y)) + c, ay = fabs(hfa::quo_keep(hv, h, y)) + c;
  sx = ax > sx ? ax : sx;
  sy = ay > sy ? ay : sy;
  return true;
}

}  // namespace hf
