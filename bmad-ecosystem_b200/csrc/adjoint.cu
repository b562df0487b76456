// adjoint.cu -- d(loss)/d(element strengths) on the GPU (bmadgpu_loss_grad of include/bmadgpu.h).
//
// A particle's turns follow one another, forward and in reverse, and a few thousand particles do not
// fill the chip: with one thread per particle the sweep is bound by the latency of a single warp
// (4096 particles, 451 elements, 32 turns: 158 ms). Only what is serial by nature is left that way:
//   k_adj_forward  one thread per particle: the turns, storing the state at the start of each turn
//                  (or, above kTurnStore, of every `every`-th, re-run by segment in reverse);
//   k_adj_inputs   one thread per (turn, particle): re-runs the turn, storing every element's input;
//   k_adj_turnjac  one thread per (turn, particle): the reverse sweep with the seven unit cotangents,
//                  i.e. the turn's Jacobian J^T;
//   k_adj_chain    one thread per particle: lambda_t = J_t^T lambda_(t+1), 49 products a turn, storing
//                  the cotangent at the end of each turn;
//   k_adj_grad     one thread per (turn, particle): the reverse sweep with that cotangent, writing the
//                  strength derivatives of the turn;
//   k_adj_collect  adds them to each particle's [slot] column, last turn first.
// Turns go through these in chunks from the last to the first, sized by kChunkBytes; where the memory for
// that is not there, in smaller chunks, from `every`-spaced checkpoints, and at last one turn of a part of
// the particles (a slab) at a time (AdjPlan). No atomics and a fixed order of every sum, so the result
// depends neither on scheduling nor on `every`, the chunks or the slabs.
// k_adj_reduce: one CTA per slot sums the column in a fixed order (deterministic), divides by the
// strength (scale form -> d/dk) and writes the gradient; slot n_slot sums the loss.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "adjoint.cuh"
#include "capi_internal.h"
#include "particle.cuh"

using namespace bmadgpu;

namespace bmadgpu {
cudaError_t adjoint_upload_constants();
}

namespace {

constexpr int kAdjBlock = 64;
constexpr size_t kTurnStore = (size_t)1 << 30;   // turn starts kept for the whole run up to this size
constexpr size_t kChunkBytes = (size_t)2 << 30;  // element inputs, Jacobians and derivatives of a chunk of turns

struct AdjArgs {
  const EleHdr* hdr;
  const ApRec* ap;
  const double* pool;
  int32_t n_ele;
  int64_t N;                 // particles: stride of the per-particle buffers
  Globals G;
  const int32_t* param_of_ele;  // [n_ele]: gradient slot of the element, -1 if none
  int32_t n_slot;
  double* vec;               // [6][N] in/out
  double* beta;              // [N] in/out
  int32_t* state;            // [N] in/out
  double* turns;             // [rows][7][N]: states at turn starts
  // a chunk of n_t turns of the particles [j0, j0 + n_j): NT = n_t n_j threads, thread t n_j + q is particle
  // j0 + q in turn row t of the chunk
  int64_t NT, j0, n_j;
  double* inputs;            // [n_ele][7][NT]
  double* jac;               // [7][7][NT]: row c, the image of unit cotangent c
  double* lam_end;           // [7][NT]: cotangent at the end of the turn
  double* part;              // [n_slot][NT]; null: a chunk is one turn, added to gradbuf at once
  double* lam;               // [7][N]: cotangent at the start of the chunk's first turn
  double* gradbuf;           // [n_slot][N]
  double* lossbuf;           // [N]
  double loss_scale;
};

__device__ __forceinline__ void put7(double* q, int64_t stride, const Particle& p) {
  q[0] = p.x;
  q[stride] = p.px;
  q[2 * stride] = p.y;
  q[3 * stride] = p.py;
  q[4 * stride] = p.z;
  q[5 * stride] = p.pz;
  q[6 * stride] = p.beta;
}
__device__ __forceinline__ void get7(const double* q, int64_t stride, Particle& p) {
  p.x = q[0];
  p.px = q[stride];
  p.y = q[2 * stride];
  p.py = q[3 * stride];
  p.z = q[4 * stride];
  p.pz = q[5 * stride];
  p.beta = q[6 * stride];
  p.state = S_ALIVE;
}

// Turns [t0, t0 + n_t) of every particle that is alive, from its vec/beta (from_vec) or from turns row
// row_in; before turn t (every `every`-th of the run) the state goes to turns row row0 + (t - t0) / every.
// The state after the last turn returns to vec/beta/state when from_vec is set. REF: the reference's element
// order, for lattices that track in it (Globals::hi_hot_pz = 0).
template <bool REF>
__global__ void __launch_bounds__(kAdjBlock) k_adj_forward(const __grid_constant__ AdjArgs a, int t0, int n_t, int every,
                                                           int row0, int row_in, int from_vec) {
  const int64_t j = (int64_t)blockIdx.x * kAdjBlock + threadIdx.x;
  if (j >= a.N || a.state[j] != S_ALIVE) return;
  const int64_t N = a.N;
  Particle p;
  if (from_vec) {
    p.x = a.vec[j];
    p.px = a.vec[N + j];
    p.y = a.vec[2 * N + j];
    p.py = a.vec[3 * N + j];
    p.z = a.vec[4 * N + j];
    p.pz = a.vec[5 * N + j];
    p.beta = a.beta[j];
    p.state = S_ALIVE;
  } else {
    get7(a.turns + (int64_t)row_in * 7 * N + j, N, p);
  }
  refresh_particle(p, a.G);
  LossInfo li;
  bool alive = true;
  for (int t = 0; t < n_t && alive; ++t) {
    if (t % every == 0) put7(a.turns + (int64_t)(row0 + t / every) * 7 * N + j, N, p);
    alive = track_turn<false, REF>(p, a.hdr, a.pool, a.ap, a.G, 0, a.n_ele, t0 + t == 0, t0 + t, li);
  }
  if (!from_vec) return;
  a.vec[j] = p.x;
  a.vec[N + j] = p.px;
  a.vec[2 * N + j] = p.y;
  a.vec[3 * N + j] = p.py;
  a.vec[4 * N + j] = p.z;
  a.vec[5 * N + j] = p.pz;
  a.beta[j] = p.beta;
  a.state[j] = p.state;
}

// Loss and its cotangent: sum over particles alive after the run of loss_scale (x^2 + y^2).
__global__ void k_adj_loss(const __grid_constant__ AdjArgs a) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.N) return;
  const bool alive = a.state[j] == S_ALIVE;  // lost particles are outside the loss
  const double x = a.vec[j], y = a.vec[2 * a.N + j];
  a.lossbuf[j] = alive ? a.loss_scale * (x * x + y * y) : 0.0;
  for (int k = 0; k < 7; k++) a.lam[k * a.N + j] = 0;
  if (alive) {
    a.lam[j] = 2 * a.loss_scale * x;
    a.lam[2 * a.N + j] = 2 * a.loss_scale * y;
  }
}

// Row row0 + t of turns is the start of the chunk's turn t; first: it is the run's first turn.
template <bool REF>
__global__ void __launch_bounds__(128) k_adj_inputs(const __grid_constant__ AdjArgs a, int row0, int first) {
  const int64_t i = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (i >= a.NT) return;
  const int64_t t = i / a.n_j, j = a.j0 + i - t * a.n_j;
  if (a.state[j] != S_ALIVE) return;
  Particle p;
  get7(a.turns + (row0 + t) * 7 * a.N + j, a.N, p);
  refresh_particle(p, a.G);
  LossInfo li;
  for (int ie = 0; ie < a.n_ele; ++ie) {
    put7(a.inputs + (int64_t)ie * 7 * a.NT + i, a.NT, p);
    track_turn<false, REF>(p, a.hdr, a.pool, a.ap, a.G, ie, ie + 1, first && t == 0 && ie == 0, 0, li);
  }
}

// The reverse sweep of one turn over its elements, cotangents a[NC]; GRAD: derivatives to part.
template <int NC, bool GRAD>
__device__ __forceinline__ void turn_sweep(const AdjArgs& A, int64_t i, int64_t j, Adj (&a)[NC]) {
  AdjCache k;
  double pz = 0, beta = 0;
  bool have = false;
  Particle next;
  get7(A.inputs + (int64_t)(A.n_ele - 1) * 7 * A.NT + i, A.NT, next);
  for (int ie = A.n_ele - 1; ie >= 0; --ie) {
    Particle p = next;
    if (ie > 0) get7(A.inputs + (int64_t)(ie - 1) * 7 * A.NT + i, A.NT, next);  // arrives during this element
    if (!have || p.pz != pz || p.beta != beta) {
      refresh(p, A.G);
      k = adj_caches(p, A.G);
      pz = p.pz;
      beta = p.beta;
      have = true;
    }
    double gs[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) gs[c] = 0;
    const EleHdr& h = A.hdr[ie];
    if (h.kind == K_RFCAV || h.n_step > 1) refresh(p, A.G);  // the bodies that are re-run on the way
    else p.e_factor = k.ef;
    vjp_element<NC>(h, A.pool, p, k, a, gs, A.G);
    if (GRAD) {
      const int slot = A.param_of_ele[ie];
      if (slot >= 0) {
        if (A.part) A.part[(int64_t)slot * A.NT + i] = gs[0];
        else A.gradbuf[(int64_t)slot * A.N + j] += gs[0];
      }
    }
  }
}

__global__ void __launch_bounds__(128) k_adj_turnjac(const __grid_constant__ AdjArgs A) {
  const int64_t i = (int64_t)blockIdx.x * 128 + threadIdx.x, j = A.j0 + i % A.n_j;
  if (i >= A.NT || A.state[j] != S_ALIVE) return;
  Adj a[7];
#pragma unroll
  for (int c = 0; c < 7; c++)
    a[c] = Adj{c == 0 ? 1.0 : 0.0, c == 1 ? 1.0 : 0.0, c == 2 ? 1.0 : 0.0, c == 3 ? 1.0 : 0.0,
               c == 4 ? 1.0 : 0.0, c == 5 ? 1.0 : 0.0, c == 6 ? 1.0 : 0.0};
  turn_sweep<7, false>(A, i, j, a);
#pragma unroll
  for (int c = 0; c < 7; c++) {
    double* q = A.jac + (int64_t)c * 7 * A.NT + i;
    q[0] = a[c].x;
    q[A.NT] = a[c].px;
    q[2 * A.NT] = a[c].y;
    q[3 * A.NT] = a[c].py;
    q[4 * A.NT] = a[c].z;
    q[5 * A.NT] = a[c].pz;
    q[6 * A.NT] = a[c].beta;
  }
}

__global__ void __launch_bounds__(kAdjBlock) k_adj_chain(const __grid_constant__ AdjArgs A, int n_t) {
  const int64_t q = (int64_t)blockIdx.x * kAdjBlock + threadIdx.x, j = A.j0 + q;
  if (q >= A.n_j || A.state[j] != S_ALIVE) return;
  double l[7];
#pragma unroll
  for (int k = 0; k < 7; k++) l[k] = A.lam[k * A.N + j];
  const int64_t NT = A.NT, n_j = A.n_j;
  const double* __restrict__ jac = A.jac + q;
  double* __restrict__ lam_end = A.lam_end + q;
  for (int t = n_t - 1; t >= 0; --t) {
    const int64_t i = t * n_j;
    double m[49];
#pragma unroll
    for (int k = 0; k < 49; k++) m[k] = jac[(int64_t)k * NT + i];
#pragma unroll
    for (int k = 0; k < 7; k++) lam_end[k * NT + i] = l[k];
    double s[7];
#pragma unroll
    for (int k = 0; k < 7; k++) {
      s[k] = 0;
#pragma unroll
      for (int c = 0; c < 7; c++) s[k] += l[c] * m[c * 7 + k];
    }
#pragma unroll
    for (int k = 0; k < 7; k++) l[k] = s[k];
  }
#pragma unroll
  for (int k = 0; k < 7; k++) A.lam[k * A.N + j] = l[k];
}

__global__ void __launch_bounds__(128) k_adj_grad(const __grid_constant__ AdjArgs A) {
  const int64_t i = (int64_t)blockIdx.x * 128 + threadIdx.x, j = A.j0 + i % A.n_j;
  if (i >= A.NT || A.state[j] != S_ALIVE) return;
  const double* q = A.lam_end + i;
  Adj a[1] = {Adj{q[0], q[A.NT], q[2 * A.NT], q[3 * A.NT], q[4 * A.NT], q[5 * A.NT], q[6 * A.NT]}};
  turn_sweep<1, true>(A, i, j, a);
}

// Of a chunk of several turns, which holds all particles (j0 = 0, n_j = N).
__global__ void __launch_bounds__(128) k_adj_collect(const __grid_constant__ AdjArgs A, int n_t, int slot0) {
  const int64_t j = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (j >= A.N || A.state[j] != S_ALIVE) return;
  const int64_t s = slot0 + blockIdx.y;
  double g = A.gradbuf[s * A.N + j];
#pragma unroll 8
  for (int t = n_t - 1; t >= 0; --t) g += A.part[s * A.NT + t * A.N + j];
  A.gradbuf[s * A.N + j] = g;
}

// Sum of row r of a [rows][N] buffer in a fixed order; one CTA of 256 threads per row.
__global__ void k_adj_reduce(const double* __restrict__ gradbuf, const double* __restrict__ lossbuf, int64_t N,
                             int n_slot, const double* __restrict__ strength, double* __restrict__ out) {
  __shared__ double part[256];
  const int r = blockIdx.x;
  const double* row = r < n_slot ? gradbuf + (int64_t)r * N : lossbuf;
  double s = 0;
  for (int64_t j = threadIdx.x; j < N; j += 256) s += row[j];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[r] = r < n_slot ? part[0] / strength[r] : part[0];
}

}  // namespace

namespace bmadgpu {

cudaError_t adjoint_upload_constants() {
  double cm[22][22], cf[22][22];
  build_cmulti_tables(cm, cf);
  cudaError_t e = cudaMemcpyToSymbol(c_cmulti, cm, sizeof(cm));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_cfull, cf, sizeof(cf));
}

}  // namespace bmadgpu

namespace {

// How the turns and particles of one call are divided. Turn starts: all of them where they fit (whole: one
// segment of all turns), so that nothing is run twice; else the checkpoints of segments of `every` turns and,
// after them, the turn starts of the segment in hand. chunk: turns of a chunk; slab: particles of a chunk of
// one turn, all of them unless memory is short.
struct AdjPlan {
  bool whole;
  int32_t seg, chunk;
  int64_t slab;
};
constexpr int64_t kMinSlab = 32;

// Device buffers of one call, carved from one block of the context's scratch.
struct AdjBuffers {
  size_t used = 0;
  unsigned char* base = nullptr;  // null while the sizes are added up
  template <class T>
  void get(T** p, size_t count) {
    if (base) *p = reinterpret_cast<T*>(base + used);
    used += (count * sizeof(T) + 255) & ~(size_t)255;
  }
};

// Strength attribute of an element the gradient is taken for, or 0 if it is not a strength
// element; all of the element's field coefficients must scale with it.
int strength_of(const bmadgpu_element& e, double* k, std::string& why) {
  switch (e.key) {
    case BMADGPU_QUADRUPOLE: *k = e.k1; break;
    case BMADGPU_SEXTUPOLE: *k = e.k2; break;
    case BMADGPU_OCTUPOLE: *k = e.k3; break;
    default: why = "gradient element is not a quadrupole, sextupole or octupole"; return BMADGPU_EINVAL;
  }
  if (*k == 0) {
    why = "gradient element has zero strength (the derivative is taken in scale form)";
    return BMADGPU_EINVAL;
  }
  if (e.hkick != 0 || e.vkick != 0) {
    why = "gradient element has hkick/vkick, which do not scale with its strength";
    return BMADGPU_EUNSUPPORTED;
  }
  if (!e.scale_multipoles) {
    for (int n = 0; n < BMADGPU_N_POLE; n++)
      if (e.a_pole[n] != 0 || e.b_pole[n] != 0) {
        why = "gradient element has multipoles not scaled with its strength (scale_multipoles = F)";
        return BMADGPU_EUNSUPPORTED;
      }
  }
  return BMADGPU_OK;
}

}  // namespace

extern "C" int bmadgpu_loss_grad(bmadgpu_ctx* c, const bmadgpu_lattice* lat, const bmadgpu_bunch* b, int32_t n_turns,
                                 int32_t every, int32_t n_param, const int32_t* param_ele, double* loss,
                                 double* grad) {
  if (!c || !lat || !b || !loss || (n_param > 0 && (!param_ele || !grad))) return fail(BMADGPU_EINVAL, "NULL argument");
  if (b->n < 1 || !b->vec || !b->beta || !b->state) return fail(BMADGPU_EINVAL, "bunch is empty or incomplete");
  if (n_turns < 1 || every < 1 || n_param < 0) return fail(BMADGPU_EINVAL, "bad turn count, interval or parameter count");
  if (lat->device != c->device) return fail(BMADGPU_EINVAL, "lattice and context are on different devices");
  const int32_t n_ele = (int32_t)lat->pk.info.n_ele;
  const EleHdr* hdr = reinterpret_cast<const EleHdr*>(lat->pk.image.data());
  for (int32_t i = 0; i < n_ele; i++)
    if (adj_supported(hdr[i]))
      return fail(BMADGPU_EUNSUPPORTED, "element " + std::to_string(i) +
                                            " is outside the adjoint path (edge fringe, bend k1 or multipoles, thin "
                                            "multipole, pitch or z_offset, or more than 16 steps)");
  std::vector<int32_t> slot_of(n_ele, -1);
  std::vector<double> strength(n_param);
  for (int32_t s = 0; s < n_param; s++) {
    const int32_t i = param_ele[s];
    if (i < 0 || i >= n_ele) return fail(BMADGPU_EINVAL, "gradient element index out of range");
    if (slot_of[i] >= 0) return fail(BMADGPU_EINVAL, "gradient element listed twice");
    std::string why;
    int r = strength_of(lat->eles[i], &strength[s], why);
    if (r) return fail(r, why + " (element " + std::to_string(i) + ")");
    slot_of[i] = s;
  }
  CUDA_TRY(cudaSetDevice(c->device));
  const int64_t N = b->n;
  const size_t slots = (size_t)(n_param > 0 ? n_param : 1);
  AdjPlan plan;
  plan.whole = (size_t)N * 56 * (size_t)n_turns <= kTurnStore;
  plan.seg = plan.whole ? n_turns : std::min(every, n_turns);
  const size_t per_turn = (size_t)N * 8 * ((size_t)n_ele * 7 + 49 + 7 + slots);
  // one wave of the Jacobian kernel (256 threads per SM), whose time a part of a second wave would double
  const size_t wave = std::max<size_t>(1, (size_t)c->sm_count * 256 / (size_t)N);
  plan.chunk = (int32_t)std::max<size_t>(1, std::min({kChunkBytes / per_turn, (size_t)plan.seg, wave}));
  plan.slab = N;
  double *d_vec, *d_beta, *d_turn, *d_ele, *d_jac, *d_lam_end, *d_part, *d_lam, *d_grad, *d_loss, *d_strength, *d_out;
  int32_t *d_state, *d_slot;
  Workspace work(c);
  AdjBuffers buf;
  auto lay_out = [&]() {
    const size_t CN = (size_t)plan.chunk * (size_t)plan.slab;
    const size_t n_seg = (size_t)((n_turns + plan.seg - 1) / plan.seg);
    buf.used = 0;
    buf.get(&d_vec, 6 * N);
    buf.get(&d_beta, N);
    buf.get(&d_state, N);
    buf.get(&d_turn, (plan.whole ? (size_t)plan.seg : n_seg + plan.seg) * 7 * N);
    buf.get(&d_ele, (size_t)n_ele * 7 * CN);
    buf.get(&d_jac, 49 * CN);
    buf.get(&d_lam_end, 7 * CN);
    buf.get(&d_part, plan.chunk > 1 ? slots * CN : 1);
    buf.get(&d_lam, 7 * (size_t)N);
    buf.get(&d_grad, slots * N);
    buf.get(&d_loss, N);
    buf.get(&d_strength, slots);
    buf.get(&d_out, slots + 1);
    buf.get(&d_slot, (size_t)n_ele);
  };
  for (lay_out(); !work.get(buf.used); lay_out()) {
    if (plan.chunk > 1) {
      plan.chunk /= 2;
    } else if (plan.whole && (n_turns + every - 1) / every + every < n_turns) {
      plan.whole = false;
      plan.seg = every;
    } else if (plan.slab > kMinSlab) {
      plan.slab = std::max<int64_t>(kMinSlab, (plan.slab / 2 + 31) / 32 * 32);
    } else {
      return fail(BMADGPU_ENOMEM, "cannot allocate the adjoint's device buffers");
    }
  }
  buf.base = static_cast<unsigned char*>(work.ptr);
  lay_out();
  const bool whole = plan.whole;
  const int32_t seg = plan.seg, n_seg = (n_turns + seg - 1) / seg, chunk = plan.chunk;
  cudaStream_t s = c->stream;
  CUDA_TRY(cudaMemcpyAsync(d_vec, b->vec, 6 * N * sizeof(double), cudaMemcpyHostToDevice, s));
  CUDA_TRY(cudaMemcpyAsync(d_beta, b->beta, N * sizeof(double), cudaMemcpyHostToDevice, s));
  CUDA_TRY(cudaMemcpyAsync(d_state, b->state, N * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  CUDA_TRY(cudaMemcpyAsync(d_slot, slot_of.data(), n_ele * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  if (n_param > 0)
    CUDA_TRY(cudaMemcpyAsync(d_strength, strength.data(), n_param * sizeof(double), cudaMemcpyHostToDevice, s));
  CUDA_TRY(cudaMemsetAsync(d_grad, 0, slots * N * sizeof(double), s));
  AdjArgs a;
  std::memset(&a, 0, sizeof(a));
  a.hdr = reinterpret_cast<const EleHdr*>(lat->d_table);
  a.ap = reinterpret_cast<const ApRec*>(lat->d_table + lat->pk.info.hdr_bytes);
  a.pool = reinterpret_cast<const double*>(lat->d_table + lat->pk.info.hdr_bytes + lat->pk.info.ap_bytes);
  a.n_ele = n_ele;
  a.N = N;
  a.G = lat->G;
  a.param_of_ele = d_slot;
  a.n_slot = n_param;
  a.vec = d_vec;
  a.beta = d_beta;
  a.state = d_state;
  a.turns = d_turn;
  a.inputs = d_ele;
  a.jac = d_jac;
  a.lam_end = d_lam_end;
  a.part = chunk > 1 ? d_part : nullptr;
  a.lam = d_lam;
  a.gradbuf = d_grad;
  a.lossbuf = d_loss;
  a.loss_scale = 1.0 / (double)N;
  const unsigned grid = (unsigned)((N + kAdjBlock - 1) / kAdjBlock);
#if defined(BG_FAST_MAPS)
  const bool ref = a.G.hi_hot_pz == 0;
  const auto forward = ref ? k_adj_forward<true> : k_adj_forward<false>;
  const auto inputs = ref ? k_adj_inputs<true> : k_adj_inputs<false>;
#else
  const auto forward = k_adj_forward<false>;
  const auto inputs = k_adj_inputs<false>;
#endif
  forward<<<grid, kAdjBlock, 0, s>>>(a, 0, n_turns, whole ? 1 : seg, 0, 0, 1);
  k_adj_loss<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(a);
  c->launches += 2;
  for (int32_t g = n_seg - 1; g >= 0; --g) {
    const int32_t t0 = g * seg, nt = std::min(seg, n_turns - t0);
    const int32_t row0 = whole ? 0 : n_seg;
    if (!whole) {
      forward<<<grid, kAdjBlock, 0, s>>>(a, t0, nt, 1, row0, g, 0);
      c->launches++;
    }
    for (int32_t end = nt; end > 0;) {
      const int32_t begin = std::max(0, end - chunk), n = end - begin;
      for (a.j0 = 0; a.j0 < N; a.j0 += plan.slab) {
        a.n_j = std::min(plan.slab, N - a.j0);
        a.NT = (int64_t)n * a.n_j;
        const unsigned wide = (unsigned)((a.NT + 127) / 128);
        inputs<<<wide, 128, 0, s>>>(a, row0 + begin, t0 + begin == 0);
        k_adj_turnjac<<<wide, 128, 0, s>>>(a);
        k_adj_chain<<<(unsigned)((a.n_j + kAdjBlock - 1) / kAdjBlock), kAdjBlock, 0, s>>>(a, n);
        k_adj_grad<<<wide, 128, 0, s>>>(a);
        c->launches += 4;
      }
      for (int32_t s0 = 0; a.part && s0 < n_param; s0 += 32768) {
        const dim3 all((unsigned)((N + 127) / 128), (unsigned)std::min(n_param - s0, 32768));
        k_adj_collect<<<all, 128, 0, s>>>(a, n, s0);
        c->launches++;
      }
      end = begin;
    }
  }
  CUDA_TRY(cudaGetLastError());
  k_adj_reduce<<<(unsigned)(n_param + 1), 256, 0, s>>>(d_grad, d_loss, N, n_param, d_strength, d_out);
  CUDA_TRY(cudaGetLastError());
  c->launches++;
  std::vector<double> out(n_param + 1);
  CUDA_TRY(cudaMemcpyAsync(out.data(), d_out, (n_param + 1) * sizeof(double), cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  for (int32_t i = 0; i < n_param; i++) grad[i] = out[i];
  *loss = out[n_param];
  return check_err_flag(c);
}
