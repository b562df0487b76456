// fastmaps.cuh -- the element maps of the default build, for the elements rings are made of.
//
// The maps of maps.cuh follow the reference's operand order operation by operation. That order is
// what the correctly rounded build needs (bit equality with the reference's algorithm), but it costs
// five libm calls and four roots or quotients per bend, four libm calls per quadrupole and one sum
// term per order and power in a multipole kick. Here the same functions of the particle are written
// with fewer operations and explicit fused multiply-adds: 212 instructions (62 of them FP64) per element of a
// 200-cell ring with multipoles, where that order takes 714. What bounds the kernels is the number of
// instructions and the dependent chains, not the FP64 pipe.
//   - longitudinal momenta: 1 - ps/rel and rel/ps - 1 are series in e = (px^2 + py^2)/(1 + pz)^2, which
//     is below 1e-4 for every particle that stays in an aperture, so no root is taken and neither
//     quantity is formed as a difference;
//   - quadrupole: cos, sin, cosh and sinh of sqrt(|k|) L are even or odd halves of the same two
//     series in u = k L^2, so both planes come from one evaluation without a root;
//   - bend: no trigonometric function of the particle: sin and cos of (angle + phi_1) and of the
//     exit direction are components of the momentum, and the arc over its chord is a series in the
//     chord; the position's large constant terms cancel analytically, so x keeps its relative
//     precision where the reference's order subtracts numbers about 1e3 times larger;
//   - multipole kick: one Horner evaluation of sum (b_n + i a_n) (x + i y)^n;
//   - losses: integer comparisons of the coordinates' high words accept a particle that is well
//     inside every limit.
// Against the same maps in quadruple precision the results are closer than the reference's order is
// (tests/test_fastmaps_cpu.py). Every form has a stated range. A particle that is outside it anywhere
// in an element, or not well inside the limits at its end, goes through that element again in the
// reference's forms with the reference's tests (cold_track1, out of line: one call per element, so
// that the loop keeps its registers); so does every particle in the elements that have no form here.
#pragma once
#include <string.h>

#include "elements.cuh"

namespace bmadgpu {

#if defined(__CUDACC__)
BG_HD uint32_t hi_abs(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }
BG_HD int hi_word(double v) { return __double2hiint(v); }
BG_HD double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
#else
inline int hi_word(double v) {
  uint64_t u;
  memcpy(&u, &v, 8);
  return (int)(u >> 32);
}
inline uint32_t hi_abs(double v) { return (uint32_t)hi_word(v) & 0x7fffffffu; }
inline double rcp_seed(double x) { return 1.0f / (float)x; }
#endif

// The quadrupole's series 1/n! (E: 4, 8, 12, 16; O: 2, 6, 10, 14; Es: 5, 9, 13, 17; Os: 3, 7, 11, 15),
// read as operands from constant memory: as literals each would take two moves per use.
#if defined(__CUDACC__)
#define BG_SERIES __constant__
#else
#define BG_SERIES
#endif
static BG_SERIES const double c_series[16] = {
    1.0 / 24.0,      1.0 / 40320.0,   1.0 / 479001600.0,  1.0 / 20922789888000.0,
    0.5,             1.0 / 720.0,     1.0 / 3628800.0,    1.0 / 87178291200.0,
    1.0 / 120.0,     1.0 / 362880.0,  1.0 / 6227020800.0, 1.0 / 355687428096000.0,
    1.0 / 6.0,       1.0 / 5040.0,    1.0 / 39916800.0,   1.0 / 1307674368000.0};

// 1 / x for x in the normal range: the third-order Newton (Householder) step y0 (1 + e + e^2), e = 1 - x y0.
// The hardware's approximation keeps 20 bits: |e| < 2^-19.9 over 2^32 arguments, so e^3 is below 2^-59; the
// result was within 0.51 units in the last place of 1 / x there.
BG_HD double rcp_f(double x) {
  const double y = rcp_seed(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// rel/ps - 1 = 1/sqrt(1 - e) - 1 and 1 - ps/rel = 1 - sqrt(1 - e) for e < 2^-12, to e^4 (the next
// terms are below 2^-62 and 2^-65).
BG_HD double inv_root_m1(double e) {
  return e * fma(e, fma(e, fma(e, 35.0 / 128.0, 5.0 / 16.0), 3.0 / 8.0), 0.5);
}
BG_HD double one_m_root(double e) {
  return e * fma(e, fma(e, fma(e, 5.0 / 128.0, 1.0 / 16.0), 1.0 / 8.0), 0.5);
}
constexpr uint32_t kHi2m12 = 0x3f300000u;     // high word of 2^-12
constexpr uint32_t kHiQuarter = 0x3fd00000u;  // high word of 1/4
constexpr uint32_t kHiHalf = 0x3fe00000u;     // of 1/2
constexpr uint32_t kHi32 = 0x40400000u;       // of 32
constexpr uint32_t kHi2m8 = 0x3f700000u;      // of 2^-8
constexpr uint32_t kHiNano = 0x3e112e0cu;     // one above that of 1e-9

BG_HD uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }

// The cached functions of pz and beta for these maps; hot: the maps below cover this pz and beta
// (|pz| < 1/4, not NaN), and enough of the lattice's elements have a form (Globals::hi_hot_pz).
// They change only in cold_track1.
BG_HD void finish_f(Particle& p, const Globals& G) {  // from refresh()'s
  p.lez = p.lez_series ? p.pz * p.lez_a * G.lez_me2 : p.lez_a * G.inv_beta0;
  p.hot = hi_abs(p.pz) < G.hi_hot_pz && p.beta > 0;
}
BG_HD void refresh_f(Particle& p, const Globals& G) {
  refresh(p, G);
  finish_f(p, G);
}

// track1 with the reference's forms and tests. The maps that change pz or beta refresh the caches
// themselves; the low-energy term's is formed for the maps that read it.
BG_COLD int cold_track1(Particle& p, const EleHdr* __restrict__ h, const double* __restrict__ pool,
                        const ApRec* __restrict__ ap, const Globals& G, bool entry_check) {
  const double pz = p.pz, beta = p.beta;
  if (h->kind == K_QUAD || (h->flags & F_BEND_K1)) refresh_lez(p, G);
  const int loc = track1<true>(p, *h, pool, ap, G, entry_check);
  if (p.pz != pz || p.beta != beta) finish_f(p, G);
  return loc;
}

// Two entries of a parameter block at an even index (blocks are 16-byte aligned).
struct Pair {
  double a, b;
};
BG_HD Pair load2(const double* __restrict__ b) {
#if defined(__CUDACC__)
  const double2 v = *reinterpret_cast<const double2*>(b);
  return Pair{v.x, v.y};
#else
  return Pair{b[0], b[1]};
#endif
}

// The coordinates that change inside an element (pz and beta do not in these maps): a copy to work on
// where a range is tested after some of them have changed. The maps take it or the particle itself.
struct Orbit {
  double x, px, y, py, z;
};

// A map writes its result only if the particle is in the range it states, and says so.

// track_a_drift: with P = px/rel, Q = py/rel, e = P^2 + Q^2, px/ps = P (1 + v) and
// dz = L (beta/beta0 - 1 - v), v = rel/ps - 1. Range: e < 2^-12.
template <class T>
BG_HD bool drift_f(T& o, const Particle& c, double L) {
  const double P = o.px * c.e_factor, Q = o.py * c.e_factor;
  const double e = fma(P, P, Q * Q);
  if ((uint32_t)hi_word(e) >= kHi2m12) return false;  // NaN too
  const double v = inv_root_m1(e);
  const double s = fma(L, v, L);
  o.x = fma(s, P, o.x);
  o.y = fma(s, Q, o.y);
  o.z = fma(L, c.dzb - v, o.z);
  return true;
}

// One quadrupole step. b: [b1, L, step, b1/L, b1 step^2/L]. Range: |k| step^2 < 1/2.
// With u = k step^2: cos(sqrt u) = E - u O, cosh = E + u O, E and O series in u^2; likewise
// sin(sqrt u)/sqrt u and sinh(sqrt u)/sqrt u. Truncation below 2^-55 for |u| < 1/2. k < 0 (u < 0)
// exchanges the planes in the same formulas.
template <class T>
BG_HD bool quad_step_f(T& o, const Particle& q, const double* __restrict__ b) {
  const double ef = q.e_factor;
  const double u = b[4] * ef;
  if (hi_abs(u) >= kHiHalf) return false;
  const Pair lk = load2(b + 2);
  const double L = lk.a, b1l = lk.b;
  const double w = u * u;
  double E = fma(c_series[3], w, c_series[2]), O = fma(c_series[7], w, c_series[6]);
  double Es = fma(c_series[11], w, c_series[10]), Os = fma(c_series[15], w, c_series[14]);
  E = fma(E, w, c_series[1]);
  O = fma(O, w, c_series[5]);
  Es = fma(Es, w, c_series[9]);
  Os = fma(Os, w, c_series[13]);
  E = fma(E, w, c_series[0]);
  O = fma(O, w, c_series[4]);
  Es = fma(Es, w, c_series[8]);
  Os = fma(Os, w, c_series[12]);
  // deviations from the drift: cos - 1, sin/(sqrt(u) L) - 1 and their hyperbolic counterparts, so that
  // the coordinates keep their own rounding
  E = E * w;
  Es = Es * w;
  const double dcx = fma(-u, O, E), dcy = fma(u, O, E);
  const double sx = fma(L, fma(-u, Os, Es), L), sy = fma(L, fma(u, Os, Es), L);
  const double cx = 1 + dcx, cy = 1 + dcy;
  const double x = o.x, y = o.y;
  const double P = o.px * ef, Q = o.py * ef;  // px/rel, py/rel
  // z: -1/4 { k [(L - c s) x - 2 s^2 P] x + (L + c s) P^2 } in x, the same with -k in y
  const double ax = fma(-cx, sx, L), bx = fma(cx, sx, L), ay = fma(-cy, sy, L), by = fma(cy, sy, L);
  const double Ax = fma(-2 * (sx * sx), P, ax * x), Ay = fma(-2 * (sy * sy), Q, ay * y);
  const double k = b1l * ef;
  double S = k * fma(Ax, x, -(Ay * y));
  S = fma(bx * P, P, S);
  S = fma(by * Q, Q, S);
  o.z = fma(L, q.lez, fma(-0.25, S, o.z));
  o.x = x + fma(dcx, x, sx * P);
  o.px = o.px + fma(dcx, o.px, -(b1l * sx) * x);
  o.y = y + fma(dcy, y, sy * Q);
  o.py = o.py + fma(dcy, o.py, (b1l * sy) * y);
  return true;
}

// Multipole kick px -= Re S, py += Im S, S = sum_n (b_n + i a_n)(x + i y)^n; c: (b_n, a_n).
// Range: |x|, |y| < 32 (the powers stay finite).
template <int NP>
BG_HD void kick_sum(double x, double y, const double* __restrict__ c, double& re, double& im) {
  re = c[2 * (NP - 1)];  // b_n alone, n >= 2
  im = 0;
#pragma unroll
  for (int n = NP - 2; n >= 0; n--) {
    const double t = n >= 2 ? fma(re, x, fma(-im, y, c[2 * n])) : fma(re, x, -(im * y));
    im = fma(re, y, im * x);
    re = t;
  }
}
BG_HD bool kicks_f(Orbit& o, const double* __restrict__ c, int np, bool b_from2) {
  const double x = o.x, y = o.y;
  if (umax(hi_abs(x), hi_abs(y)) >= kHi32) return false;
  double re, im;
  switch (b_from2 ? np : 0) {  // unrolled: the loads' latency is off the chain
    case 3: kick_sum<3>(x, y, c, re, im); break;
    case 4: kick_sum<4>(x, y, c, re, im); break;
    case 5: kick_sum<5>(x, y, c, re, im); break;
    case 6: kick_sum<6>(x, y, c, re, im); break;
    case 7: kick_sum<7>(x, y, c, re, im); break;
    case 8: kick_sum<8>(x, y, c, re, im); break;
    case 9: kick_sum<9>(x, y, c, re, im); break;
    case 10: kick_sum<10>(x, y, c, re, im); break;
    case 11: kick_sum<11>(x, y, c, re, im); break;
    default:
      re = c[2 * (np - 1)];
      im = c[2 * (np - 1) + 1];
#pragma unroll 2
      for (int n = np - 2; n >= 0; n--) {
        const double t = fma(re, x, fma(-im, y, c[2 * n]));
        im = fma(re, y, fma(im, x, c[2 * n + 1]));
        re = t;
      }
      break;
  }
  o.px = o.px - re;
  o.py = o.py + im;
  return true;
}
// The same for a sextupole alone: S = b_2 (x + i y)^2.
template <class T>
BG_HD void kick2_f(T& o, double b2) {
  o.px = fma(-b2, fma(o.x, o.x, -(o.y * o.y)), o.px);
  o.py = fma(2 * b2, o.x * o.y, o.py);
}

BG_HD void tilt_f(Orbit& o, double c, double s) {
  const double x = o.x, px = o.px;
  o.x = fma(c, x, s * o.y);
  o.y = fma(c, o.y, -s * x);
  o.px = fma(c, px, s * o.py);
  o.py = fma(c, o.py, -s * px);
}
// offset_particle without pitches; m: [x_off, y_off, cos_t, sin_t].
BG_HD void offset_set_f(Orbit& o, const double* __restrict__ m, bool has_tilt) {
  o.x = o.x - m[0];
  o.y = o.y - m[1];
  if (has_tilt) tilt_f(o, m[2], m[3]);
}
BG_HD void offset_unset_f(Orbit& o, const double* __restrict__ m, bool has_tilt) {
  if (has_tilt) tilt_f(o, m[2], -m[3]);
  o.x = o.x + m[0];
  o.y = o.y + m[1];
}

// offset_particle with pitches, z_offset or a misaligned bend's frame; m: one side of the frame block.
// The position's steps are one affine map here; the longitudinal momentum is rel (1 - one_m_root), and
// the drift to the edge, without reference motion, as in drift_f (none below 1e-14, as the reference).
BG_HD bool frame_f(Orbit& o, const Particle& q, const double* __restrict__ m) {
  const double rel = 1 + q.pz, ef = q.e_factor;
  double P = o.px * ef, Q = o.py * ef;
  const double e1 = fma(P, P, Q * Q);
  const double ps = fma(-rel, one_m_root(e1), rel);
  const double nx = fma(m[0], o.x, fma(m[1], o.y, m[2])), ny = fma(m[3], o.x, fma(m[4], o.y, m[5]));
  const double s = fma(m[6], o.x, fma(m[7], o.y, m[8]));
  const double px = fma(m[9], o.px, fma(m[10], o.py, m[11] * ps)), py = fma(m[12], o.px, fma(m[13], o.py, m[14] * ps));
  P = px * ef;
  Q = py * ef;
  const double e2 = fma(P, P, Q * Q);
  if (umax((uint32_t)hi_word(e1), (uint32_t)hi_word(e2)) >= kHi2m12) return false;
  const double ds = fabs(s) > 1e-14 ? s : 0.0;
  const double l = fma(ds, inv_root_m1(e2), ds);
  o.x = fma(l, P, nx);
  o.y = fma(l, Q, ny);
  o.z = o.z - l;
  o.px = px;
  o.py = py;
  return true;
}

// hwang_bend_edge_kick for upright faces without a fringe integral or field index: only the gs2
// terms are left, gs2 = g_tot.
template <class T>
BG_HD void upright_edge_f(T& o, double ef, double g) {
  const double h = 0.5 * g * ef, yy = o.y * o.y, q = h * o.px;
  o.z = fma(-(q * ef), yy, o.z);
  o.py = fma(-2 * q, o.y, o.py);
  o.x = fma(h, yy, o.x);
}

// hwang_bend_edge_kick in full; e: the edge's coefficients (table.h).
template <class T>
BG_HD void hwang_edge_f(T& o, double ef, const double* __restrict__ e, bool entering) {
  const double gt = e[0], gt2 = e[1], gs2 = e[2], k1t = e[3], fg = e[4], gtot = e[5], cdpx = e[6];
  const double sg = entering ? 1.0 : -1.0;
  const double v1 = o.x, v2 = o.px, v3 = o.y, v4 = o.py;
  const double v11 = v1 * v1, v33 = v3 * v3, v13 = v1 * v3;
  const double dx = (0.5 * sg * ef) * fma(gs2, v33, -(gt2 * v11));
  const double a = fma(v1, v2, -(v3 * v4)), b = k1t * (v11 - v33);
  const double dpx = ef * (entering ? fma(0.5 * cdpx, v33, fma(gt2, a, b))
                                    : fma(-gt2, a, fma(-0.5 * (gt * gt2), v11 + v33, b)));
  const double c = fma(gt2 * v1, v4, ((gtot + gt2) * v2) * v3);
  const double dpy = ef * fma(fg, v3, fma(-sg, c, (entering ? -2 * k1t : fma(gt, gs2, -2 * k1t)) * v13));
  double s = fma(v33, fg, (v11 * v1) * (fma(-gt, gt2, 4.0 * k1t) * (1.0 / 6.0)));
  s = fma(0.5 * fma(gt, gs2, -4.0 * k1t) * v1, v33, s);
  s = fma(sg, fma(gt2, fma(v11, v2, -2.0 * (v13 * v4)), -((v2 * v33) * gs2)), s);
  o.z = fma(0.5 * (ef * ef), s, o.z);
  o.x = v1 + dx;
  o.px = v2 + fma(gt, v1, dpx);
  o.y = fma(sg * gt2 * ef, v13, v3);
  o.py = v4 + fma(-gt, v3, dpy);
}

// Exact sector bend step. The momentum along the rotated axes is Sp = sa ps + ca px =
// pt sin(angle + phi_1), Cp = ca ps - sa px; the exit px is Sp - g_tot h, h = (1 + g x) L sinc, and
// R = sqrt(pt^2 - px_exit^2). The reference's xi = alpha / (rad + cos_plus) is h N / D with
// N = Sp + px_exit, D = R + Cp, and its value on the design orbit, xi0 = h0 sa / (1 + ca), is
// L^2 g cosc; the difference is dxi = h0 [dN + g x N - tan(angle/2) dD] / D with dN, dD the
// deviations of N and D from it.
// The chord L_c, L_c^2 = (xi0 + dxi)^2 + (h0 + x sa)^2, gives half the bending angle,
// sin(hp) = g_tot L_c / (2 pt), and the arc L_p = L_c F(q), F(q) = asin(s)/s at q = s^2 = sin(hp)^2.
// Chord and F are taken as deviations from the design chord L_c0 and from F(q0), q0 = (g_tot L_c0/2)^2,
// the latter by its Taylor series at q0 (the table's coefficients): the path's difference from the
// design length, about 1e-4 of it, is not formed by subtracting the two.
// beta L / beta0 is rounded as the reference rounds it: that rounding is the same in every bend of a
// turn, so it is the one term whose last bit shows in z against the reference's tracking.
// Range: a step length above zero (fast_header), the chord and the arc being positive;
// the momentum series' e < 2^-12 at both ends; L_c^2/L_c0^2 - 1 and q - q0 below 2^-8, where
// their series, truncated at the sixth power, are good to 2^-58; clear of the reference's semi-linear
// map near the zero orbit (track_a_bend.f90:136-159, all of |px|, |py|, |pz| < 1e-9).
template <class T>
BG_HD bool bend_step_f(T& o, const Particle& q, const double* __restrict__ b, const Globals& G, bool has_dg) {
  const Pair gl = load2(b + SB_F), cs = load2(b + SB_F + 2), ht = load2(b + SB_F + 4), xh = load2(b + SB_F + 6);
  const double g = gl.a, L = gl.b, ca = cs.a, sa = cs.b, h0 = ht.a;
  const double x = o.x, px = o.px, py = o.py, pz = q.pz, ef = q.e_factor;
  const double rel = 1 + pz;
  const double P = px * ef, Q = py * ef, e3 = Q * Q, e1 = fma(P, P, e3);
  const double d = fma(-rel, one_m_root(e1), pz);  // ps - 1
  const double gx = g * x;
  const double dS = fma(ca, px, sa * d);
  double pxf = fma(-sa, gx, dS);
  if (has_dg) pxf = fma(-(b[3] * h0), 1 + gx, pxf);
  const double Pf = pxf * ef, e2 = fma(Pf, Pf, e3);
  const double dR = fma(-rel, one_m_root(e2), pz);  // R - 1
  const double dC = fma(ca, d, -(sa * px));
  const double dN = dS + pxf, N = sa + dN;
  const double dD = dR + dC;
  const double E = fma(gx, N, fma(-ht.b, dD, dN));
  const double dxi = (h0 * E) * rcp_f((1 + ca) + dD);
  const double t = sa * x;
  const double W = fma(dxi, xh.a + dxi, t * (xh.b + t));  // L_c^2 - L_c0^2
  const Pair ic = load2(b + SB_F + 8), gc = load2(b + SB_F + 10), fa = load2(b + SB_F + 12), fb = load2(b + SB_F + 14),
             fc = load2(b + SB_F + 16), fd = load2(b + SB_F + 18);
  const double del = W * ic.a;       // over L_c0^2
  const double v = inv_root_m1(e3);  // rel/pt - 1
  const double ipt = fma(ef, v, ef);
  // q - q0, with pt^2 - 1 = pz (2 + pz) - py^2
  const double dq = (gc.a * (ipt * ipt)) * fma(-ic.b, fma(pz, 2 + pz, -(py * py)), W);
  const double xf = fma(ca, x, dxi);
  // the comparisons of high words compare values: all of them are non-negative, and NaN is above
  const uint32_t mom = umax(umax(hi_abs(px), hi_abs(py)), hi_abs(pz));
  if ((umax((uint32_t)hi_word(e1), (uint32_t)hi_word(e2)) >= kHi2m12) | (umax(hi_abs(del), hi_abs(dq)) >= kHi2m8) |
      (mom < kHiNano) | (hi_abs(xf) >= G.hi_max_ap))
    return false;
  double c = fma(del, -21.0 / 1024.0, 7.0 / 256.0);
  c = fma(c, del, -5.0 / 128.0);
  c = fma(c, del, 1.0 / 16.0);
  c = fma(c, del, -1.0 / 8.0);
  c = fma(c, del, 0.5);
  const double Lc0 = gc.b;
  const double dLc = Lc0 * (c * del);
  double f = fma(fd.a, dq, fc.b);
  f = fma(f, dq, fc.a);
  f = fma(f, dq, fb.b);
  f = fma(f, dq, fb.a);
  f = fma(f, dq, fa.b);
  const double dLp = fma(Lc0 + dLc, f * dq, fma(dLc, fa.a, fd.b));
  const double Lp = L + dLp;
  const double bl = q.beta * L, bq = bl * G.inv_beta0;
  const double bL = fma(fma(-G.beta0, bq, bl), G.inv_beta0, bq);  // beta L / beta0, correctly rounded (div_rcp)
  o.x = xf;
  o.px = pxf;
  o.y = fma(Lp, fma(Q, v, Q), o.y);
  o.z = o.z + (((bL - L) - dLp) - Lp * v);
  return true;
}

// An element with a form (FastHdr f). Returns false, with the particle as it was, if the particle is
// outside a range inside the element.
BG_HD bool element_f(Particle& p, const EleHdr* __restrict__ h, const FastHdr& f, const double* __restrict__ pool,
                     const Globals& G) {
  const double* b = pool + f.param;
  const uint32_t c = f.code;
  const bool mis = c & FC_MISALIGN, tilted = c & FC_TILT;
  if ((c & FC_ENTRANCE) && !((hi_abs(p.x) < f.acc_x) & (hi_abs(p.y) < f.acc_y))) return false;
  if (!(c & (FC_MISALIGN | FC_PITCH))) {  // nothing moves before the range is tested: in place
    switch (c & FC_BODY) {
      case FC_DRIFT: return drift_f(p, p, b[0]);
      case FC_QUAD: return quad_step_f(p, p, b);
      case FC_BEND:
        if (c & FC_EDGE_IN) break;
        if (!bend_step_f(p, p, b, G, c & FC_DG)) return false;
        if (c & FC_EDGE_OUT) {
          if (c & FC_UPRIGHT) upright_edge_f(p, p.e_factor, -b[2]);
          else hwang_edge_f(p, p.e_factor, b + SB_EDGE_OUT, false);
        }
        return true;
      default: break;
    }
  }
  Orbit o = {p.x, p.px, p.y, p.py, p.z};
  // misalign of a pitched quadrupole or thick multipole
  const int m = tilted && (c & FC_PITCH)
                    ? (h->kind == K_QUAD ? QD_FIXED : TH_FIXED) + kick_doubles(h->n_pole, h->n_step) : 0;
  if (c & FC_PITCH) {
    if (!frame_f(o, p, pool + h->extra)) return false;
    if (tilted) tilt_f(o, b[m + 2], b[m + 3]);
  }
  switch (c & FC_BODY) {
    case FC_DRIFT:
      if (!drift_f(o, p, b[0])) return false;
      break;
    case FC_QUAD:  // one step, no kicks; misalign after the block
      if (mis) offset_set_f(o, b + QD_FIXED, tilted);
      if (!quad_step_f(o, p, b)) return false;
      if (mis) offset_unset_f(o, b + QD_FIXED, tilted);
      break;
    case FC_SEXT: {  // one step between two equal kicks of order 2
      const Pair lb = load2(b);
      if (mis) offset_set_f(o, b + TH_FIXED + 6, tilted);
      kick2_f(o, lb.b);
      if (!drift_f(o, p, lb.a)) return false;
      kick2_f(o, lb.b);
      if (mis) offset_unset_f(o, b + TH_FIXED + 6, tilted);
      break;
    }
    case FC_BEND:
      if (mis) tilt_f(o, b[SB_FIXED + 2], b[SB_FIXED + 3]);  // ref_tilt
      if (c & FC_EDGE_IN) {
        if (c & FC_UPRIGHT) upright_edge_f(o, p.e_factor, b[2]);
        else hwang_edge_f(o, p.e_factor, b + SB_EDGE_IN, true);
      }
      // orbit_too_large after the edge; the step's own range covers the momenta
      if ((c & (FC_EDGE_IN | FC_MISALIGN | FC_PITCH)) && umax(hi_abs(o.x), hi_abs(o.y)) >= G.hi_max_ap) return false;
      if (!bend_step_f(o, p, b, G, c & FC_DG)) return false;
      if (c & FC_EDGE_OUT) {
        if (c & FC_UPRIGHT) upright_edge_f(o, p.e_factor, -b[2]);
        else hwang_edge_f(o, p.e_factor, b + SB_EDGE_OUT, false);
      }
      if (mis) tilt_f(o, b[SB_FIXED + 2], -b[SB_FIXED + 3]);
      break;
    case FC_STEPS: {  // quadrupole or thick multipole of any steps and kicks
      const int np = h->n_pole, n_step = h->n_step;
      const bool quad = h->kind == K_QUAD, from2 = h->flags & F_KICK_B_FROM2;
      const double* k = b + (quad ? QD_FIXED : TH_FIXED);
      const double* ml = k + kick_doubles(np, n_step);
      if (mis) offset_set_f(o, ml, tilted);
      for (int i = 0; i <= n_step; i++) {
        if (i > 0)
          if (!(quad ? quad_step_f(o, p, b) : drift_f(o, p, b[0]))) return false;
        if (np && !kicks_f(o, (i == 0 || i == n_step) ? k : k + 2 * np, np, from2)) return false;
      }
      if (mis) offset_unset_f(o, ml, tilted);
      break;
    }
    default:  // FC_MARKER
      break;
  }
  if (c & FC_PITCH) {
    if (tilted) tilt_f(o, b[m + 2], -b[m + 3]);
    if (!frame_f(o, p, pool + h->extra + 18)) return false;
  }
  p.x = o.x;
  p.px = o.px;
  p.y = o.y;
  p.py = o.py;
  p.z = o.z;
  return true;
}

// The tests after an element's body (track1.f90:289-329), as track1 makes them.
BG_COLD int cold_exit(Particle& p, const EleHdr* __restrict__ h, const ApRec* __restrict__ ap, const Globals& G) {
  if (orbit_too_large(p, G)) return L_UPSTREAM;
  if (h->flags & F_AP_EXIT) {
    aperture(p, ap[h->ap_index], h->flags & F_AP_ELLIPTICAL, h->flags & F_AP_WINDOW);
    if (p.state != S_ALIVE) return L_DOWNSTREAM;
  }
  return 0;
}

// Whether the launch's first element may go through track1_f's forms: the entrance orbit_too_large
// test would pass.
BG_HD bool entry_f(const Particle& p, const Globals& G) {
  return (umax(hi_abs(p.x), hi_abs(p.y)) < G.hi_max_ap) & (umax(hi_abs(p.px), hi_abs(p.py)) < kHiQuarter);
}

// track1. Returns coord%location of a loss, or 0. p.hot: the forms cover the particle's pz (refresh_f)
// and, at the first element of a launch, its entrance coordinates (entry_f).
BG_HD int track1_f(Particle& p, const EleHdr* __restrict__ h, const FastHdr& f, const double* __restrict__ pool,
                   const ApRec* __restrict__ ap, const Globals& G, bool entry_check) {
  if (p.hot && (f.code & FC_BODY) != FC_COLD) {
    if (element_f(p, h, f, pool, G)) {
      // with |px|, |py|, |pz| < 1/4 no test of the momenta finds a loss
      if ((hi_abs(p.x) < f.acc_x) & (hi_abs(p.y) < f.acc_y) & (umax(hi_abs(p.px), hi_abs(p.py)) < kHiQuarter)) return 0;
      Particle q;
      q.x = p.x; q.px = p.px; q.y = p.y; q.py = p.py; q.z = p.z; q.pz = p.pz; q.state = p.state;
      const int loc = cold_exit(q, h, ap, G);
      p.state = q.state;
      return loc;
    }
  }
  Particle q = p;
  const int loc = cold_track1(q, h, pool, ap, G, entry_check);
  p = q;
  return loc;
}

}  // namespace bmadgpu
