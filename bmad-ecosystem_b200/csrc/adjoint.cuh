// adjoint.cuh -- hand-written reverse-mode derivatives (vector-Jacobian products) of the element
// maps in maps.cuh / elements.cuh, for d(loss)/d(element strengths).
//
// State: (x, px, y, py, z, pz, beta). beta is carried as a coordinate of its own because the
// maps use the tracked coord%beta (exact bend z, energy kick, RF time, low-energy z), not a
// function of pz. Each vjp_* takes the primitive's INPUT particle (caches refreshed), and maps the
// cotangent of its output (Adj) to the cotangent of its input in place. Branches follow the
// forward map's branch at that input; the aperture and orbit checks are piecewise constant and
// contribute nothing. Parameter cotangents are returned as "scale" derivatives: for a set of
// coefficients c that all scale with one strength k (b1 = k1 L and the multipoles of a quadrupole;
// b_n = k_n L / n! and scaled multipoles of a sextupole/octupole), dL/dk = sum_c c dL/dc / k.
//
// The Jacobians restate, in reverse form, the make_matrix branches of the reference maps:
// track_a_drift.f90:94-114, track_a_quadrupole.f90:204-223 with quad_mat2_calc.f90:65-79,
// track_a_bend.f90:211-300, multipole_mod.f90:123-126, apply_energy_kick.f90:57-69.
#pragma once
#include "elements.cuh"

namespace bmadgpu {

struct Adj {
  double x, px, y, py, z, pz, beta;
};

// Elements with more body steps (or RF slices) than this are outside the adjoint path.
constexpr int kAdjMaxSteps = 16;

// Functions of pz (and beta) the derivatives share: they change only at an energy kick, so a sweep over
// the elements forms them once per stretch (adj_caches).
struct AdjCache {
  double ef;      // 1 / (1 + pz)
  double ddzb;    // d(dzb)/d(pz): dzb = beta(pz)/beta0 - 1, dbeta/dpz = p0c m^2 / E^3
  double lez_pz;  // d(low_energy_z)/d(pz) per unit length (series branch)
  double lez_b;   // d(low_energy_z)/d(beta) per unit length (the other branch)
};

// p: caches refreshed (refresh()).
BG_HD AdjCache adj_caches(const Particle& p, const Globals& G) {
  AdjCache c;
  c.ef = 1 / (1 + p.pz);
  const double P = G.p0c * (1 + p.pz);
  const double E2 = P * P + G.mass2;
  c.ddzb = p.beta > 0 ? G.p0c * G.mass2 / (G.beta0 * E2 * sqrt(E2)) : 0.0;
  if (p.lez_series) {
    const double dlez = -3 * G.lez_b02 / 2 + 2 * p.pz * G.lez_f;
    c.lez_pz = G.lez_me2 * (p.lez_a + p.pz * dlez);
    c.lez_b = 0;
  } else {
    c.lez_pz = 0;
    c.lez_b = 1 / G.beta0;
  }
  return c;
}

// Each primitive below forms the coefficients of its Jacobian at the input particle once and applies
// the transpose to NC cotangents: one in the gradient sweep, seven (the unit vectors) where a whole
// turn's Jacobian is wanted.

// track_a_drift
template <int NC>
BG_HD void vjp_drift(const Particle& p, const AdjCache& k, double L, Adj (&a)[NC]) {
  if (L == 0) return;
  const double ar = p.px * k.ef, br = p.py * k.ef;
  const double s2 = ar * ar + br * br;
  const double ips = 1 / sqrt(1 - s2), l = L * ips, l3 = l * ips * ips;
  const double xx = l + ar * ar * l3, xy = ar * br * l3, yy = l + br * br * l3, xz = ar * l3, yz = br * l3;
  const double zb = L * k.ddzb;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const double ab = (a[c].x * xx + a[c].y * xy - a[c].z * xz) * k.ef;
    const double bb = (a[c].x * xy + a[c].y * yy - a[c].z * yz) * k.ef;
    a[c].px += ab;
    a[c].py += bb;
    a[c].pz += a[c].z * zb - (ab * ar + bb * br);
  }
}

// cos, sin / sqrt(k) of quad_mat2_calc (quad_mat2_calc.f90:34-47) for +-k and their derivatives with
// respect to k. For |k| l^2 < 1/2 by the series in u = k l^2: c(u) = sum (-u)^n/(2n)!,
// s(u) = l sum (-u)^n/(2n+1)! for the focusing sign, u -> -u for the other.
struct QuadCs {
  double c, s, dc, ds;
};
BG_HD QuadCs quad_cs(double k, double l) {  // c'' = k c: k > 0 hyperbolic
  QuadCs q;
  const double u = k * (l * l), l2 = l * l;
  if (fabs(u) < 0.5) {
    double c = 1.0 / 20922789888000.0, s = 1.0 / 355687428096000.0, dc = 8.0 / 20922789888000.0,
           ds = 8.0 / 355687428096000.0;
    const double f[8] = {1.0, 0.5, 1.0 / 24.0, 1.0 / 720.0, 1.0 / 40320.0, 1.0 / 3628800.0, 1.0 / 479001600.0,
                         1.0 / 87178291200.0};
    const double g[8] = {1.0, 1.0 / 6.0, 1.0 / 120.0, 1.0 / 5040.0, 1.0 / 362880.0, 1.0 / 39916800.0,
                         1.0 / 6227020800.0, 1.0 / 1307674368000.0};
#pragma unroll
    for (int n = 7; n >= 0; n--) {
      c = c * u + f[n];
      s = s * u + g[n];
      if (n > 0) {
        dc = dc * u + n * f[n];
        ds = ds * u + n * g[n];
      }
    }
    q.c = c;
    q.s = s * l;
    q.dc = dc * l2;
    q.ds = ds * l2 * l;
    return q;
  }
  const double sk = sqrt(fabs(k)), skl = sk * l;
  if (k < 0) {
    q.c = cos(skl);
    q.s = sin(skl) / sk;
  } else {
    q.c = cosh(skl);
    q.s = sinh(skl) / sk;
  }
  q.dc = l * q.s / 2;
  q.ds = (l * q.c - q.s) / (2 * k);
  return q;
}

// One plane of a quadrupole step with k (quad_mat2_calc's), at (x, px): cotangents of k and rel as
// coefficients of the cotangents of the plane's x', px' and of z'.
struct QuadPlane {
  double m11, m12, m21;      // m22 = m11
  double zx, zp;             // dz/dx, dz/dpx
  double kx, kp, kz;         // d/dk of x', px', z'
  double rx, rp, rz;         // d/drel of the same
};
BG_HD QuadPlane quad_plane(double k, double l, double rel, double ef, double x, double px) {
  const QuadCs q = quad_cs(k, l);
  QuadPlane o;
  o.m11 = q.c;
  o.m12 = q.s * ef;
  o.m21 = k * q.s * rel;
  const double cs = q.c * q.s, dcs = q.dc * q.s + q.c * q.ds, s2 = q.s * q.s;
  const double z0 = k * (l - cs) / 4, z1 = -k * s2 * ef / 2, z2 = -(cs + l) * ef * ef / 4;
  o.zx = 2 * z0 * x + z1 * px;
  o.zp = z1 * x + 2 * z2 * px;
  o.kx = x * q.dc + px * q.ds * ef;
  o.kp = px * q.dc + x * (q.s + k * q.ds) * rel;
  o.kz = x * x * ((l - cs) / 4 - k * dcs / 4) - x * px * (s2 + 2 * k * q.s * q.ds) * ef / 2 -
         px * px * dcs * ef * ef / 4;
  o.rx = -px * q.s * ef * ef;
  o.rp = x * k * q.s;
  o.rz = -(x * px * z1 + 2 * px * px * z2) * ef;
  return o;
}

// One quad body step (quad_step); gscale += d/d(b1) contribution times b1 (scale form).
template <int NC>
BG_HD void vjp_quad_step(const Particle& p, const AdjCache& k, double b1, double length, double sl, Adj (&a)[NC],
                         double (&gscale)[NC]) {
  const double rel = 1 + p.pz;
  const double k1 = b1 / length * k.ef;
  const QuadPlane X = quad_plane(-k1, sl, rel, k.ef, p.x, p.px), Y = quad_plane(k1, sl, rel, k.ef, p.y, p.py);
  const double lp = sl * k.lez_pz, lb = sl * k.lez_b;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const Adj o = a[c];
    const double gk1 = (o.y * Y.kx + o.py * Y.kp + o.z * Y.kz) - (o.x * X.kx + o.px * X.kp + o.z * X.kz);
    const double gr = (o.x * X.rx + o.px * X.rp + o.z * X.rz) + (o.y * Y.rx + o.py * Y.rp + o.z * Y.rz);
    a[c].x = o.x * X.m11 + o.px * X.m21 + o.z * X.zx;
    a[c].px = o.x * X.m12 + o.px * X.m11 + o.z * X.zp;
    a[c].y = o.y * Y.m11 + o.py * Y.m21 + o.z * Y.zx;
    a[c].py = o.y * Y.m12 + o.py * Y.m11 + o.z * Y.zp;
    a[c].pz += gr - gk1 * k1 * k.ef + o.z * lp;
    a[c].beta += o.z * lb;
    gscale[c] += gk1 * k1;  // k1 is proportional to b1: b1 dL/db1 = k1 dL/dk1
  }
}

// ab_multipole_kicks with pre-scaled coefficients c = (b_n, a_n): px += kx, py += ky with
// kx - i ky = -S, S = sum (b_n + i a_n)(x + i y)^n, by Horner with its derivative.
template <int NC>
BG_HD void vjp_ab_kicks(const Particle& p, const double* __restrict__ c, int n_pole, Adj (&a)[NC],
                        double (&gscale)[NC]) {
  const double x = p.x, y = p.y;
  double re = 0, im = 0, dr = 0, di = 0;
  for (int n = n_pole - 1; n >= 0; n--) {
    const double td = dr * x - di * y + re;
    di = dr * y + di * x + im;
    dr = td;
    const double t = re * x - im * y + c[2 * n];
    im = re * y + im * x + c[2 * n + 1];
    re = t;
  }
#pragma unroll
  for (int i = 0; i < NC; i++) {
    gscale[i] += a[i].py * im - a[i].px * re;
    const double gx = a[i].py * di - a[i].px * dr, gy = a[i].px * di + a[i].py * dr;
    a[i].x += gx;
    a[i].y += gy;
  }
}

// tilt (rotation by (c, s)); the inverse rotation passes -s.
template <int NC>
BG_HD void vjp_tilt(double c, double s, Adj (&a)[NC]) {
#pragma unroll
  for (int i = 0; i < NC; i++) {
    const double ax = a[i].x, ay = a[i].y, apx = a[i].px, apy = a[i].py;
    a[i].x = c * ax - s * ay;
    a[i].y = s * ax + c * ay;
    a[i].px = c * apx - s * apy;
    a[i].py = s * apx + c * apy;
  }
}

// Exact sbend body step in the trigonometric variables of bend_exact_step itself, one cotangent: for bends
// with F_BEND_LONG (negative lengths, whose arc goes the long way round, and angles whose half asin may not
// give).
BG_COLD void vjp_bend_trig(const Particle& p, const double* __restrict__ b, Adj& a, const Globals& G) {
  double l = b[0], g = b[1], g_tot = b[2], dg = b[3], angle = b[4];
  double cos_a = b[5], sin_a = b[6], sinc_a = b[7], cosc_a = b[8], gl2_sincc = b[9];
  double x = p.x, px = p.px, py = p.py, pz = p.pz;
  double rel = 1 + pz;
  if (dg == 0 && fabs(x * g) < 1e-9 && fabs(px) < 1e-9 && fabs(py) < 1e-9 && fabs(pz) < 1e-9) {
    double rpp = rel * G.p0c;
    double den = rpp * rpp + G.mass2;
    double gam2 = G.mass2 / den;
    double m56 = l * (gam2 - gl2_sincc);
    double dm56 = l * (-G.mass2 * 2 * rpp * G.p0c / (den * den));
    Adj o = a;
    a.x = o.x * cos_a + o.px * (-g * sin_a) + o.z * (-g * l * sinc_a);
    a.px = o.x * l * sinc_a + o.px * cos_a + o.z * (-g * l * l * cosc_a);
    a.py = o.py + o.y * l;
    a.pz = o.pz + o.x * g * l * l * cosc_a + o.px * g * l * sinc_a + o.z * (m56 + dm56 * pz);
    return;
  }
  // forward intermediates
  double pt = sqrt(rel * rel - py * py);
  double g_p = g_tot / pt;
  double u = px / pt;
  double phi_1 = asin(u);
  double cp = cos(angle + phi_1), sp = sin(angle + phi_1);
  double gx1 = 1 + g * x;
  double ls = gx1 * l * sinc_a;
  double alpha = 2 * gx1 * sp * l * sinc_a - g_p * (ls * ls);
  double r = cp * cp + g_p * alpha;
  double rad = sqrt(r);
  double xi, den = 0;
  if (cp > 0) {
    den = rad + cp;
    xi = alpha / den;
  } else {
    xi = (rad - cp) / g_p;
  }
  double L_u = xi;
  double L_v = -1 * (l * sinc_a + x * sin_a);
  double L_c = sqrt(L_v * L_v + L_u * L_u);
  double theta = atan2(L_u, -L_v);
  double angle_p = 2 * (angle + phi_1 - theta);
  double hp = angle_p / 2;
  double S = 1, dS = 0;
  if (fabs(hp) >= 1e-8) {
    S = sin(hp) / hp;
    dS = (hp * cos(hp) - sin(hp)) / (hp * hp);
  }
  double L_p = L_c / S;
  double psi = phi_1 + angle - angle_p;
  // reverse sweep
  double b_pt = 0, b_rel = 0, b_Lp = 0, b_phi = 0, b_angp = 0, b_Lc = 0, b_Lu = 0, b_Lv = 0, b_xi = 0;
  double b_alpha = 0, b_rad = 0, b_cp = 0, b_sp = 0, b_gp = 0, b_gx1 = 0, b_ls = 0;
  double b_x = 0, b_px = 0, b_py = 0;
  // z' = z + beta l / beta0 - rel L_p / pt
  double beta_bar = a.beta + a.z * l / G.beta0;
  b_rel += -a.z * L_p / pt;
  b_Lp += -a.z * rel / pt;
  b_pt += a.z * rel * L_p / (pt * pt);
  // y' = y + py L_p / pt
  b_py += a.y * L_p / pt;
  b_Lp += a.y * py / pt;
  b_pt += -a.y * py * L_p / (pt * pt);
  // px' = pt sin(psi)
  b_pt += a.px * sin(psi);
  double b_psi = a.px * pt * cos(psi);
  b_phi += b_psi;
  b_angp += -b_psi;
  // py' = py, pz' = pz
  b_py += a.py;
  double b_pz = a.pz;
  // L_p = L_c / S(hp)
  b_Lc += b_Lp / S;
  double b_S = -b_Lp * L_c / (S * S);
  b_angp += b_S * dS / 2;
  // angle_p = 2 (angle + phi_1 - theta)
  b_phi += 2 * b_angp;
  double b_theta = -2 * b_angp;
  double X = -L_v, Y = L_u, R2 = X * X + Y * Y;
  b_Lu += b_theta * X / R2;
  double b_X = -b_theta * Y / R2;
  b_Lv += -b_X;
  // L_c = sqrt(L_v^2 + L_u^2)
  b_Lv += b_Lc * L_v / L_c;
  b_Lu += b_Lc * L_u / L_c;
  // L_v = -(l sinc_a + x sin_a), L_u = xi
  b_x += -b_Lv * sin_a;
  b_xi += b_Lu;
  // x' = x cos_a - l^2 g cosc_a + xi
  b_x += a.x * cos_a;
  b_xi += a.x;
  // xi
  if (cp > 0) {
    b_alpha += b_xi / den;
    double b_den = -b_xi * alpha / (den * den);
    b_rad += b_den;
    b_cp += b_den;
  } else {
    b_rad += b_xi / g_p;
    b_cp += -b_xi / g_p;
    b_gp += -b_xi * (rad - cp) / (g_p * g_p);
  }
  // rad = sqrt(r); r = cp^2 + g_p alpha
  double b_r = b_rad / (2 * rad);
  b_cp += b_r * 2 * cp;
  b_gp += b_r * alpha;
  b_alpha += b_r * g_p;
  // alpha = 2 gx1 sp l sinc_a - g_p ls^2; ls = gx1 l sinc_a
  b_gx1 += b_alpha * 2 * sp * l * sinc_a;
  b_sp += b_alpha * 2 * gx1 * l * sinc_a;
  b_gp += -b_alpha * ls * ls;
  b_ls += -b_alpha * g_p * 2 * ls;
  b_gx1 += b_ls * l * sinc_a;
  b_x += b_gx1 * g;
  // cp, sp of angle + phi_1
  b_phi += -b_cp * sp + b_sp * cp;
  // phi_1 = asin(px/pt)
  double b_u = b_phi / sqrt(1 - u * u);
  b_px += b_u / pt;
  b_pt += -b_u * px / (pt * pt);
  // g_p = g_tot / pt
  b_pt += -b_gp * g_tot / (pt * pt);
  // pt = sqrt(rel^2 - py^2)
  b_rel += b_pt * rel / pt;
  b_py += -b_pt * py / pt;
  b_pz += b_rel;
  a.x = b_x;
  a.px = b_px;
  a.py = b_py;
  a.pz = b_pz;
  a.beta = beta_bar;
  // a.y and a.z pass through (y' = y + ..., z' = z + ...)
}

// Exact sbend body step (bend_exact_step). In the momentum components of the rotated axes (Sp, Cp) and
// the exit components (pxf, R) the map has no trigonometric function of the particle but the arc over
// its chord, L_p = L_c F(q), F = asin(s)/s, q = s^2 = (g_tot L_c / 2 pt)^2:
//   pxf = ca px + sa ps - g_tot h, h = (1 + g x) L sinc, xi = h (2 pxf + g_tot h) / (R + Cp),
//   x' = x ca + xi - const, y' = y + py L_p / pt, z' = z + beta L / beta0 - rel L_p / pt.
// Four directions (x, px, py, rel) are differentiated through it. For bends without F_BEND_LONG: told apart by
// the element, not by the particle, since a test of the half angle and a call in here cost every bend (4096
// particles, 451 elements, 32 turns: 17.9 ms a gradient against 17.4).
template <int NC>
BG_HD void vjp_bend_exact(const Particle& p, const AdjCache& k, const double* __restrict__ b, Adj (&a)[NC],
                          const Globals& G) {
  const double l = b[0], g = b[1], g_tot = b[2], dg = b[3];
  const double ca = b[5], sa = b[6], sinc_a = b[7], cosc_a = b[8], gl2_sincc = b[9];
  const double x = p.x, px = p.px, py = p.py, pz = p.pz;
  const double rel = 1 + pz;
  if (dg == 0 && fabs(x * g) < 1e-9 && fabs(px) < 1e-9 && fabs(py) < 1e-9 && fabs(pz) < 1e-9) {
    const double rpp = rel * G.p0c;
    const double den = rpp * rpp + G.mass2;
    const double gam2 = G.mass2 / den;
    const double m56 = l * (gam2 - gl2_sincc);
    const double dm56 = l * (-G.mass2 * 2 * rpp * G.p0c / (den * den));
#pragma unroll
    for (int i = 0; i < NC; i++) {
      const Adj o = a[i];
      a[i].x = o.x * ca + o.px * (-g * sa) + o.z * (-g * l * sinc_a);
      a[i].px = o.x * l * sinc_a + o.px * ca + o.z * (-g * l * l * cosc_a);
      a[i].py = o.py + o.y * l;
      a[i].pz = o.pz + o.x * g * l * l * cosc_a + o.px * g * l * sinc_a + o.z * (m56 + dm56 * pz);
    }
    return;
  }
  const double pt2 = rel * rel - py * py;
  const double ps = sqrt(pt2 - px * px), ips = 1 / ps;
  const double ipt = 1 / sqrt(pt2);
  const double h0 = l * sinc_a, h = h0 * (1 + g * x);
  const double pxf = ca * px + sa * ps - g_tot * h;
  const double R = sqrt(pt2 - pxf * pxf), iR = 1 / R;
  const double Cp = ca * ps - sa * px;
  const double N = 2 * pxf + g_tot * h;
  const bool fwd = Cp > 0;
  const double iD = fwd ? 1 / (R + Cp) : 1 / g_tot;
  const double xi = fwd ? h * N * iD : (R - Cp) * iD;
  const double Lv = h0 + x * sa;
  const double Lc = sqrt(xi * xi + Lv * Lv), iLc = 1 / Lc;
  const double s = 0.5 * g_tot * Lc * ipt, q = s * s;
  double F, dF;  // F and dF/dq
  if (q < 0.0078125) {
    F = 1 + q * (1.0 / 6 + q * (3.0 / 40 + q * (5.0 / 112 + q * (35.0 / 1152 + q * (63.0 / 2816 +
            q * (231.0 / 13312 + q * (143.0 / 10240)))))));
    dF = 1.0 / 6 + q * (3.0 / 20 + q * (15.0 / 112 + q * (35.0 / 288 + q * (315.0 / 2816 + q * (693.0 / 6656 +
            q * (1001.0 / 10240))))));
  } else {
    // half the bending angle, beyond a right angle where the chord shortens again
    double hp = asin(fmin(fabs(s), 1.0));
    const double ct = Cp * Lv + (pxf + g_tot * h) * xi;  // sign of cos(angle + phi_1 - theta)
    if (ct < 0) hp = kPi - hp;
    F = hp / fabs(s);
    dF = (1 / cos(hp) - F) / (2 * q);
  }
  const double Lp = Lc * F, w = Lp * ipt;
  // directions: x, px, py, rel
  const double d_ps[4] = {0, -px * ips, -py * ips, rel * ips};
  const double d_pt2[4] = {0, 0, -py, rel};  // d(pt^2)/2
  double jx[4], jp[4], jy[4], jz[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double dh = i == 0 ? h0 * g : 0.0, dpx = i == 1 ? 1.0 : 0.0;
    const double dpxf = ca * dpx + sa * d_ps[i] - g_tot * dh;
    const double dR = (d_pt2[i] - pxf * dpxf) * iR;
    const double dCp = ca * d_ps[i] - sa * dpx;
    const double dxi = fwd ? (dh * N + h * (2 * dpxf + g_tot * dh) - xi * (dR + dCp)) * iD : (dR - dCp) * iD;
    const double dLc = (xi * dxi + (i == 0 ? Lv * sa : 0.0)) * iLc;
    const double dpt = d_pt2[i] * ipt * ipt;  // over pt
    const double dLp = dLc * F + Lc * dF * (2 * q) * (dLc * iLc - dpt);
    const double dw = dLp * ipt - w * dpt;
    jx[i] = (i == 0 ? ca : 0.0) + dxi;
    jp[i] = dpxf;
    jy[i] = py * dw + (i == 2 ? w : 0.0);
    jz[i] = -rel * dw - (i == 3 ? w : 0.0);
  }
  const double zb = l / G.beta0;
#pragma unroll
  for (int i = 0; i < NC; i++) {
    const Adj o = a[i];
    a[i].x = o.x * jx[0] + o.px * jp[0] + o.y * jy[0] + o.z * jz[0];
    a[i].px = o.x * jx[1] + o.px * jp[1] + o.y * jy[1] + o.z * jz[1];
    a[i].py = o.py + o.x * jx[2] + o.px * jp[2] + o.y * jy[2] + o.z * jz[2];
    a[i].pz = o.pz + o.x * jx[3] + o.px * jp[3] + o.y * jy[3] + o.z * jz[3];
    a[i].beta = o.beta + o.z * zb;
  }
}

// apply_energy_kick: (pz, beta, z) with energy gain dE; g_dE receives dL/d(dE).
BG_HD void vjp_energy_kick(const Particle& p, double dE, Adj& a, double& g_dE, const Globals& G) {
  double p0c = G.p0c;
  double rel = 1 + p.pz;
  double pc = rel * p0c;
  double beta = p.beta;
  double E_old = pc / beta;
  double E_new = E_old + dE;
  double A = (2 * E_old * dE + dE * dE) / (pc * pc);
  double S = sqrt(1 + A);
  double pz_new = p.pz + rel * sqrt_one(A);
  double pc_new = p0c * (1 + pz_new);
  double beta_new = pc_new / E_new;
  // z' = z beta_new / beta
  double b_z = a.z * beta_new / beta;
  double b_bnew = a.beta + a.z * p.z / beta;
  double b_beta = -a.z * p.z * beta_new / (beta * beta);
  // beta_new = p0c (1 + pz_new) / E_new
  double b_pznew = a.pz + b_bnew * p0c / E_new;
  double b_Enew = -b_bnew * beta_new / E_new;
  // 1 + pz_new = rel S(A), A(E_old, dE, pc)
  double b_rel = b_pznew * S;
  double b_A = b_pznew * rel / (2 * S);
  double b_Eold = b_A * 2 * dE / (pc * pc) + b_Enew;
  double b_dE = b_A * 2 * E_new / (pc * pc) + b_Enew;
  double b_pc = b_A * (-2 * A / pc);
  // E_old = pc / beta
  b_pc += b_Eold / beta;
  b_beta += -b_Eold * pc / (beta * beta);
  b_rel += b_pc * p0c;
  a.z = b_z;
  a.pz = b_rel;
  a.beta = b_beta;
  g_dE += b_dE;
}

// Tape of sub-step inputs inside one element.
struct AdjTape {
  Particle in[2 * kAdjMaxSteps + 6];
  int n = 0;
  BG_HD void push(const Particle& p) { in[n++] = p; }
};

#if defined(__CUDACC__)
#define BG_HOST_DEVICE __host__ __device__ inline
#else
#define BG_HOST_DEVICE inline
#endif

// Which element bodies the adjoint covers (elements.cuh forms). 0 if supported.
BG_HOST_DEVICE int adj_supported(const EleHdr& h) {
  if (h.flags & (F_PITCH | F_EXTRA)) return 1;  // pitched / bend-frame misalignment, electric
                                                // multipoles, higher-order edges: no
                                                // vector-Jacobian product written
  switch (h.kind) {
    case K_MARKER:
    case K_DRIFT:
      return 0;
    case K_QUAD:
    case K_THICK:
      return h.n_step <= kAdjMaxSteps ? 0 : 1;
    case K_SBEND:
      if (h.flags & (F_EDGE_IN | F_EDGE_OUT | F_BEND_K1)) return 1;
      if (h.n_pole) return 1;
      return h.n_step <= kAdjMaxSteps ? 0 : 1;
    case K_RFCAV:
      return h.n_step <= kAdjMaxSteps ? 0 : 1;
    default:
      return 1;  // thin multipoles
  }
}

// Reverse of the RF cavity body (body_rf) for one cotangent.
BG_COLD void vjp_rf(const EleHdr& h, const double* __restrict__ b, const Particle& pin, Adj& a1, double& gs1,
                    const Globals& G) {
  Adj a[1] = {a1};
  double gscale[1] = {gs1};
  Particle p = pin;
  const int np = h.n_pole;
  const double* kh = b + RF_FIXED;
  const double* mis = kh + 2 * np;
  const bool has_t = h.flags & F_TILT, misal = h.flags & F_MISALIGN;
  const double voltage = b[0], f = b[1], slice_len = b[4];
  const int n_slice = h.n_step;
  if (misal) offset_set(p, mis, has_t);
  Particle pk0 = p;  // before the entrance kicks
  if (np) ab_kicks(p, kh, np);
  const Particle p_ph = p;  // the phase is taken here
  double phase = rf_phase(p, b[2], f, b[3]);
  // forward slices: K[i] = state before kick i, D[i] = state before drift i, phases
  Particle Kin[kAdjMaxSteps + 1], Din[kAdjMaxSteps];
  double ph[kAdjMaxSteps + 1];
  for (int i = 0; i <= n_slice; i++) {
    ph[i] = phase;
    Kin[i] = p;
    double dE = 1.0 * voltage * sin(phase) / n_slice;
    if (i == 0 || i == n_slice) dE = dE / 2;
    energy_kick(p, dE, G);
    if (i != n_slice) {
      refresh(p, G);
      Din[i] = p;
      double z = p.z;
      drift(p, slice_len);
      phase = phase + kTwoPi * f * (p.z - z) / (kCLight * p.beta);
    }
  }
  refresh(p, G);
  const Particle p_exit = p;  // before the exit kicks
  if (misal && has_t) vjp_tilt<1>(mis[2], -mis[3], a);
  if (np) vjp_ab_kicks<1>(p_exit, kh, np, a, gscale);
  double b_phase = 0;
  for (int i = n_slice; i >= 0; i--) {
    if (i != n_slice) {
      // phase_{i+1} = phase_i + 2 pi f (z_after - z_before) / (c beta), beta of Din[i]
      const Particle& d = Din[i];
      Particle e = d;
      drift(e, slice_len);
      double cfac = kTwoPi * f / (kCLight * d.beta);
      a[0].z += b_phase * cfac;                // through z_after (the drift's output)
      vjp_drift<1>(d, adj_caches(d, G), slice_len, a);
      a[0].z += -b_phase * cfac;               // z_before
      a[0].beta += -b_phase * cfac * (e.z - d.z) / d.beta;
    }
    double dE = 1.0 * voltage * sin(ph[i]) / n_slice;
    double dEfac = 1.0 * voltage / n_slice;
    if (i == 0 || i == n_slice) {
      dE = dE / 2;
      dEfac = dEfac / 2;
    }
    double g_dE = 0;
    vjp_energy_kick(Kin[i], dE, a[0], g_dE, G);
    b_phase += g_dE * dEfac * cos(ph[i]);
  }
  // phase0 = modulo2(2 pi (phi0 - t f) + ..., pi), t = -z / (beta c)
  double dt_dz = -1 / (p_ph.beta * kCLight), dt_dbeta = p_ph.z / (p_ph.beta * p_ph.beta * kCLight);
  a[0].z += b_phase * (-kTwoPi * f) * dt_dz;
  a[0].beta += b_phase * (-kTwoPi * f) * dt_dbeta;
  if (np) vjp_ab_kicks<1>(pk0, kh, np, a, gscale);
  if (misal && has_t) vjp_tilt<1>(mis[2], mis[3], a);
  a1 = a[0];
  gs1 = gscale[0];
}

// Reverse of a body of several steps (quadrupole, thick multipole, bend), its sub-step inputs on a tape.
template <int NC>
BG_COLD void vjp_steps(const EleHdr& h, const double* __restrict__ b, const Particle& pin, const AdjCache& k,
                       Adj* __restrict__ ap, double* __restrict__ gp, const Globals& G) {
  Adj a[NC];
  double gscale[NC];
  for (int c = 0; c < NC; c++) {
    a[c] = ap[c];
    gscale[c] = gp[c];
  }
  Particle p = pin;
  const int np = h.n_pole, n_step = h.n_step;
  const bool quad = h.kind == K_QUAD, bend = h.kind == K_SBEND;
  const double* kh = b + (quad ? QD_FIXED : TH_FIXED);
  const double* kf = kh + 2 * np;
  const double* mis = bend ? b + SB_FIXED : kh + kick_doubles(np, n_step);
  const bool has_t = h.flags & F_TILT, misal = h.flags & F_MISALIGN;
  AdjTape t;
  if (misal) {
    if (bend) tilt(p, mis[2], mis[3]);
    else offset_set(p, mis, has_t);
  }
  for (int i = bend ? 1 : 0; i <= n_step; i++) {
    if (i > 0) {
      t.push(p);
      if (quad) quad_step(p, b[0], b[1], b[2], G);
      else if (bend && !(h.flags & F_BEND_DRIFT)) bend_exact_step(p, b, G);
      else drift(p, b[0]);
    }
    if (np) {
      t.push(p);
      ab_kicks(p, (i == 0 || i == n_step) ? kh : kf, np);
    }
  }
  if (misal && (bend || has_t)) vjp_tilt<NC>(mis[2], -mis[3], a);
  for (int i = n_step; i >= (bend ? 1 : 0); i--) {
    if (np) vjp_ab_kicks<NC>(t.in[--t.n], (i == 0 || i == n_step) ? kh : kf, np, a, gscale);
    if (i > 0) {
      const Particle& q = t.in[--t.n];
      if (quad) vjp_quad_step<NC>(q, k, b[0], b[1], b[2], a, gscale);
      else if (bend && (h.flags & F_BEND_LONG) && !(h.flags & F_BEND_DRIFT))
        for (int c = 0; c < NC; c++) vjp_bend_trig(q, b, a[c], G);
      else if (bend && !(h.flags & F_BEND_DRIFT)) vjp_bend_exact<NC>(q, k, b, a, G);
      else vjp_drift<NC>(q, k, b[0], a);
    }
  }
  if (misal && (bend || has_t)) vjp_tilt<NC>(mis[2], mis[3], a);
  for (int c = 0; c < NC; c++) {
    ap[c] = a[c];
    gp[c] = gscale[c];
  }
}

// Reverse of one element body (the part between track1's checks) at input p (caches refreshed, k its
// adj_caches): maps the cotangents of the element's output to those of its input; gscale += sum_c c dL/dc
// over the element's strength coefficients.
template <int NC>
BG_HD void vjp_element(const EleHdr& h, const double* __restrict__ pool, const Particle& pin, const AdjCache& k,
                       Adj (&a)[NC], double (&gscale)[NC], const Globals& G) {
  const double* b = pool + h.param;
  const bool misal = h.flags & F_MISALIGN, has_t = h.flags & F_TILT;
  const int np = h.n_pole;
  if (h.kind == K_DRIFT) {
    vjp_drift<NC>(pin, k, b[0], a);
  } else if (h.kind == K_QUAD && np == 0 && h.n_step == 1) {
    const double* mis = b + QD_FIXED;
    Particle p = pin;
    if (misal) offset_set(p, mis, has_t);
    if (misal && has_t) vjp_tilt<NC>(mis[2], -mis[3], a);
    vjp_quad_step<NC>(p, k, b[0], b[1], b[2], a, gscale);
    if (misal && has_t) vjp_tilt<NC>(mis[2], mis[3], a);
  } else if (h.kind == K_THICK && np > 0 && h.n_step == 1) {
    const double* kh = b + TH_FIXED;
    const double* mis = kh + kick_doubles(np, 1);
    Particle p0 = pin;
    if (misal) offset_set(p0, mis, has_t);
    Particle p1 = p0;
    ab_kicks(p1, kh, np, h.flags & F_KICK_B_FROM2);
    Particle p2 = p1;
    drift(p2, b[0]);
    if (misal && has_t) vjp_tilt<NC>(mis[2], -mis[3], a);
    vjp_ab_kicks<NC>(p2, kh, np, a, gscale);
    vjp_drift<NC>(p1, k, b[0], a);
    vjp_ab_kicks<NC>(p0, kh, np, a, gscale);
    if (misal && has_t) vjp_tilt<NC>(mis[2], mis[3], a);
  } else if (h.kind == K_SBEND && h.n_step == 1 && !misal && !(h.flags & (F_BEND_DRIFT | F_BEND_LONG))) {
    vjp_bend_exact<NC>(pin, k, b, a, G);
  } else if (h.kind == K_RFCAV) {
    for (int c = 0; c < NC; c++) vjp_rf(h, b, pin, a[c], gscale[c], G);
  } else if (h.kind != K_MARKER) {
    Adj t[NC];
    double g[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) {
      t[c] = a[c];
      g[c] = gscale[c];
    }
    vjp_steps<NC>(h, b, pin, k, t, g, G);
#pragma unroll
    for (int c = 0; c < NC; c++) {
      a[c] = t[c];
      gscale[c] = g[c];
    }
  }
}
BG_HD void vjp_element(const EleHdr& h, const double* __restrict__ pool, const Particle& pin, Adj& a, double& gscale,
                       const Globals& G) {
  Adj t[1] = {a};
  double g[1] = {gscale};
  vjp_element<1>(h, pool, pin, adj_caches(pin, G), t, g, G);
  a = t[0];
  gscale = g[0];
}

// ---- per-particle driver of the host check: forward with checkpoints, then the reverse sweep ----
// (the device spreads the same sweep over turns and particles, adjoint.cu)
#if !defined(__CUDACC__)
//
// Loss: sum over particles alive after n_turns of loss_scale * (x^2 + y^2). Buffers are
// structure-of-arrays with particle stride N: row r, component k of particle j at
// buf[(r * 7 + k) * N + j]. Checkpoints hold the state at the start of every `every`-th turn;
// in the reverse sweep each segment is re-run from its checkpoint storing the state at each turn
// start, and each turn is re-run storing every element's input, so the sweep runs backwards over
// elements with each element's input at hand (three levels: checkpoints, turns, elements).
struct AdjArgs {
  const EleHdr* hdr;
  const ApRec* ap;
  const double* pool;
  int32_t n_ele;
  int32_t n_turns;
  int32_t every;             // checkpoint interval in turns
  int64_t N;                 // particle stride of every buffer
  Globals G;
  const int32_t* param_of_ele;  // [n_ele]: gradient slot of the element, -1 if none
  double* ckpt;              // [ceil(n_turns / every)][7][N]
  double* turnbuf;           // [every][7][N]
  double* elebuf;            // [n_ele][7][N]
  double* gradbuf;           // [n_slots][N], accumulated (zeroed by the caller)
  double* lossbuf;           // [N]
  double* vec;               // [6][N] in/out
  double* beta;              // [N] in/out
  int32_t* state;            // [N] in/out
  double loss_scale;
};

BG_HD void adj_store(double* buf, int64_t row, int64_t N, int64_t j, const Particle& p) {
  double* q = buf + row * 7 * N + j;
  q[0] = p.x;
  q[N] = p.px;
  q[2 * N] = p.y;
  q[3 * N] = p.py;
  q[4 * N] = p.z;
  q[5 * N] = p.pz;
  q[6 * N] = p.beta;
}

BG_HD void adj_load(const double* buf, int64_t row, int64_t N, int64_t j, Particle& p, const Globals& G) {
  const double* q = buf + row * 7 * N + j;
  p.x = q[0];
  p.px = q[N];
  p.y = q[2 * N];
  p.py = q[3 * N];
  p.z = q[4 * N];
  p.pz = q[5 * N];
  p.beta = q[6 * N];
  p.state = S_ALIVE;
  refresh(p, G);
}

// One turn of track1 over every element; false if the particle was lost. The adjoint accepts no
// element with an extra block or a pitched offset (adj_supported), so the lean track1 serves.
BG_HD bool adj_turn(Particle& p, const AdjArgs& a, bool first_turn, double* store, int64_t j) {
  for (int ie = 0; ie < a.n_ele; ++ie) {
    if (store) adj_store(store, ie, a.N, j, p);
    if (track1<false>(p, a.hdr[ie], a.pool, a.ap, a.G, first_turn && ie == 0)) return false;
  }
  return true;
}

BG_HD void adj_particle(const AdjArgs& a, int64_t j) {
  const int64_t N = a.N;
  Particle p;
  p.x = a.vec[j];
  p.px = a.vec[N + j];
  p.y = a.vec[2 * N + j];
  p.py = a.vec[3 * N + j];
  p.z = a.vec[4 * N + j];
  p.pz = a.vec[5 * N + j];
  p.beta = a.beta[j];
  p.state = a.state[j];
  a.lossbuf[j] = 0;
  if (p.state != S_ALIVE) return;
  refresh(p, a.G);
  bool alive = true;
  for (int t = 0; t < a.n_turns && alive; ++t) {
    if (t % a.every == 0) adj_store(a.ckpt, t / a.every, N, j, p);
    alive = adj_turn(p, a, t == 0, nullptr, j);
  }
  a.vec[j] = p.x;
  a.vec[N + j] = p.px;
  a.vec[2 * N + j] = p.y;
  a.vec[3 * N + j] = p.py;
  a.vec[4 * N + j] = p.z;
  a.vec[5 * N + j] = p.pz;
  a.beta[j] = p.beta;
  a.state[j] = p.state;
  if (!alive) return;  // lost particles are outside the loss
  a.lossbuf[j] = a.loss_scale * (p.x * p.x + p.y * p.y);
  Adj lam = {2 * a.loss_scale * p.x, 0, 2 * a.loss_scale * p.y, 0, 0, 0, 0};
  const int n_seg = (a.n_turns + a.every - 1) / a.every;
  for (int seg = n_seg - 1; seg >= 0; --seg) {
    const int t0 = seg * a.every;
    const int nt = (a.n_turns - t0 < a.every) ? a.n_turns - t0 : a.every;
    Particle q;
    adj_load(a.ckpt, seg, N, j, q, a.G);
    for (int t = 0; t < nt; ++t) {
      adj_store(a.turnbuf, t, N, j, q);
      adj_turn(q, a, t0 + t == 0, nullptr, j);
    }
    for (int t = nt - 1; t >= 0; --t) {
      adj_load(a.turnbuf, t, N, j, q, a.G);
      adj_turn(q, a, t0 + t == 0, a.elebuf, j);
      for (int ie = a.n_ele - 1; ie >= 0; --ie) {
        Particle e;
        adj_load(a.elebuf, ie, N, j, e, a.G);
        double gs = 0;
        vjp_element(a.hdr[ie], a.pool, e, lam, gs, a.G);
        const int slot = a.param_of_ele[ie];
        if (slot >= 0) a.gradbuf[slot * N + j] += gs;
      }
    }
  }
}

#endif  // !__CUDACC__

}  // namespace bmadgpu
