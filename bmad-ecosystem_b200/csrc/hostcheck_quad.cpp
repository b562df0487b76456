// hostcheck_quad.cpp -- TEST-ONLY: the element maps of maps.cuh and elements.cuh in quadruple
// precision (libquadmath), the value that the rounding errors of the double-precision forms are
// measured against. The bends' trigonometric invariants are recomputed in quadruple precision.
#include <math.h>
#include <quadmath.h>
#include <stdint.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bmadgpu.h"
#include "lattice.h"
#include "table.h"

namespace bmadgpu {
typedef __float128 Q;
inline Q sqrt(Q a) { return sqrtq(a); }
inline Q fabs(Q a) { return fabsq(a); }
inline Q sin(Q a) { return sinq(a); }
inline Q cos(Q a) { return cosq(a); }
inline Q asin(Q a) { return asinq(a); }
inline Q atan2(Q a, Q b) { return atan2q(a, b); }
inline Q sinh(Q a) { return sinhq(a); }
inline Q cosh(Q a) { return coshq(a); }
inline Q exp(Q a) { return expq(a); }
inline Q tan(Q a) { return tanq(a); }
inline Q fmod(Q a, Q b) { return fmodq(a, b); }
inline Q floor(Q a) { return floorq(a); }
inline Q fma(Q a, Q b, Q c) { return fmaq(a, b, c); }
double h_cmulti_raw[22][22];
double h_cfull_raw[22][22];
}  // namespace bmadgpu

#define double bmadgpu::Q
#define BG_COUNT_OPS
#define h_cmulti h_cmulti_q
#define h_cfull h_cfull_q
#include "elements.cuh"
#undef h_cmulti
#undef h_cfull
#undef double

namespace bmadgpu {
Q h_cmulti_q[kNPole][kNPole];
Q h_cfull_q[kNPole][kNPole];
}

using namespace bmadgpu;

extern "C" {

// Tracks the bunch (host SoA) n_turns; coordinate i of particle j is hi[i n + j] + lo[i n + j].
int bmadgpu_hostcheck_quad_track(const bmadgpu_element* eles, int32_t n_ele, const bmadgpu_param* param,
                                 const bmadgpu_bunch* b, int32_t n_turns, double* hi, double* lo) {
  build_cmulti_tables(h_cmulti_raw, h_cfull_raw);
  for (int i = 0; i < kNPole; i++)
    for (int j = 0; j < kNPole; j++) {
      h_cmulti_q[i][j] = h_cmulti_raw[i][j];
      h_cfull_q[i][j] = h_cfull_raw[i][j];
    }
  PackedLattice pk;
  std::string err;
  int r = pack_lattice(eles, n_ele, *param, pk, err);
  if (r) return r;
  const uint8_t* tbl = pk.image.data();
  const EleHdr* hdr = reinterpret_cast<const EleHdr*>(tbl);
  std::vector<EleHdr> hq(hdr, hdr + n_ele);
  const ApRec* ap = reinterpret_cast<const ApRec*>(tbl + pk.info.hdr_bytes);
  const double* pd = reinterpret_cast<const double*>(tbl + pk.info.hdr_bytes + pk.info.ap_bytes);
  std::vector<Q> pool(pd, pd + pk.info.pool_doubles);
  for (const EleHdr& h : hq) {
    if (h.kind != K_SBEND) continue;
    Q* q = &pool[h.param];
    const Q L = q[0], g = q[1], a = g * L;
    if (a == 0) continue;
    q[4] = a;
    q[5] = cosq(a);
    q[6] = sinq(a);
    q[7] = sinq(a) / a;
    q[8] = 2 * sinq(a / 2) * sinq(a / 2) / (a * a);
  }
  Globals G;
  G.p0c = param->p0c; G.e_tot = param->e_tot; G.mass = param->mass; G.beta0 = param->p0c / param->e_tot;
  G.max_ap = param->max_aperture_limit; G.mass2 = param->mass * param->mass;
  double me = param->mass / param->e_tot;
  G.lez_me2 = me * me; G.lez_b02 = G.beta0 * G.beta0; G.lez_f = G.lez_b02 * (2 * G.lez_b02 - G.lez_me2 / 2);
  G.lez_thresh = 3e-7 * param->e_tot; G.charge = param->charge;
  G.inv_beta0 = 1 / G.beta0;
  const int64_t n = b->n;
  for (int64_t j = 0; j < n; j++) {
    Particle p;
    p.x = b->vec[j]; p.px = b->vec[n + j]; p.y = b->vec[2 * n + j];
    p.py = b->vec[3 * n + j]; p.z = b->vec[4 * n + j]; p.pz = b->vec[5 * n + j];
    p.beta = b->beta[j];
    p.state = b->state[j];
    refresh(p, G);
    bool lost = p.state != S_ALIVE;
    for (int turn = 0; turn < n_turns && !lost; turn++)
      for (int ie = 0; ie < n_ele && !lost; ie++)
        lost = track1(p, hq[ie], pool.data(), ap, G, turn == 0 && ie == 0) != 0;
    const Q v[6] = {p.x, p.px, p.y, p.py, p.z, p.pz};
    for (int i = 0; i < 6; i++) {
      hi[i * n + j] = (double)v[i];
      lo[i * n + j] = (double)(v[i] - hi[i * n + j]);
    }
  }
  return 0;
}

}  // extern "C"
