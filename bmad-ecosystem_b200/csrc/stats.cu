// stats.cu -- bunch statistics on the device for the long-term-tracking outputs.
//
// The sums ltt_calc_bunch_data (bsim/modules/lt_tracking_mod.f90:2369-2451) and
// calc_bunch_sigma_matrix_etc (bmad/multiparticle/beam_utils.f90:1757-1844) take over the live
// particles, in two passes as they do (the centred sums need the average first):
//   pass 1: count, sum vec_i, sum t, sum t^2, sum vec_i vec_j (i <= j)            (30 values)
//   pass 2: sum (vec_i - a_i)(vec_j - a_j) (i <= j), sum (vec_i - a_i)^3, ^4       (33 values)
// Each pass is a grid of kStatBlocks CTAs writing per-CTA partial sums (warp shuffles, then the
// warps in order) and one reduce kernel, a warp per value, that adds the partials in a fixed tree, so
// the result does not depend on scheduling. The host turns the sums into the bunch data (bunchdata.cpp).
//
// sigma_t is the root of <t^2> - <t>^2 where t is many turns long and the spread a part in 1e5 of it:
// sum t and sum t^2 are carried in double-double (Knuth's two-sum, the square exact by an FMA), so that
// the difference has the accuracy of the two rounded sums and not of the order of summation.
//
// Bound: one read of the bunch per pass (60 and 52 bytes a particle); the 592 small CTAs and loads that
// do not wait for the state keep more reads in flight, and the reduce kernel reads its partials
// coalesced instead of one thread walking 296 of them.

#include <cuda_runtime.h>

#include "stats.cuh"

namespace bmadgpu {

namespace {

constexpr int kStatThreads = 128;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// hi + lo += x (two-sum; lo gathers the rounding errors).
__device__ __forceinline__ void add_dd(double& hi, double& lo, double x) {
  const double s = hi + x;
  const double b = s - hi;
  lo += (hi - (s - b)) + (x - b);
  hi = s;
}

__device__ __forceinline__ void warp_sum_dd(double& hi, double& lo) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double h = __shfl_xor_sync(0xffffffffu, hi, o), l = __shfl_xor_sync(0xffffffffu, lo, o);
    add_dd(hi, lo, h);
    lo += l;
  }
}

// Adds the block's NV values (one per thread-local accumulator) and writes them to rows
// out[k * kStatBlocks + block].
template <int NV>
__device__ void block_sum(double (&acc)[NV], double* __restrict__ out) {
  __shared__ double part[kStatThreads / 32][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    double s = warp_sum(acc[k]);
    if (lane == 0) part[warp][k] = s;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < NV; k += kStatThreads) {
    double s = 0;
    for (int w = 0; w < kStatThreads / 32; w++) s += part[w][k];
    out[(int64_t)k * kStatBlocks + blockIdx.x] = s;
  }
}

// Double-double sum of the block to out[0] (high) and out[1] (low), rows as above.
__device__ void block_sum_dd(double hi, double lo, double* __restrict__ out_hi, double* __restrict__ out_lo) {
  __shared__ double ph[kStatThreads / 32], pl[kStatThreads / 32];
  warp_sum_dd(hi, lo);
  if ((threadIdx.x & 31) == 0) {
    ph[threadIdx.x >> 5] = hi;
    pl[threadIdx.x >> 5] = lo;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double h = 0, l = 0;
    for (int w = 0; w < kStatThreads / 32; w++) {
      add_dd(h, l, ph[w]);
      l += pl[w];
    }
    out_hi[blockIdx.x] = h;
    out_lo[blockIdx.x] = l;
  }
  __syncthreads();
}

constexpr int kRowT = 7, kRowT2 = 8;                              // rows of sum t, sum t^2
constexpr int kRowTLo = kStatPass1, kRowT2Lo = kStatPass1 + 1;    // and of their low parts

__global__ void __launch_bounds__(kStatThreads) k_stats_pass1(const double* __restrict__ vec,
                                                              const double* __restrict__ t,
                                                              const int32_t* __restrict__ state, int64_t n,
                                                              double* __restrict__ partial) {
  double acc[kStatPass1] = {0};
  double th = 0, tl = 0, qh = 0, ql = 0;
  for (int64_t j = (int64_t)blockIdx.x * kStatThreads + threadIdx.x; j < n; j += (int64_t)gridDim.x * kStatThreads) {
    // all loads first: a dead particle's are wasted, but none waits for the state
    const int32_t st = state[j];
    double v[6];
#pragma unroll
    for (int i = 0; i < 6; i++) v[i] = vec[i * n + j];
    const double tj = t ? t[j] : 0.0;
    if (st != 1) continue;
    acc[0] += 1;
#pragma unroll
    for (int i = 0; i < 6; i++) acc[1 + i] += v[i];
    add_dd(th, tl, tj);
    const double q = tj * tj;
    add_dd(qh, ql, q);
    ql += fma(tj, tj, -q);
    int k = 9;
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
      for (int m = i; m < 6; m++) acc[k++] += v[i] * v[m];
  }
  block_sum<kStatPass1>(acc, partial);
  block_sum_dd(th, tl, partial + (int64_t)kRowT * kStatBlocks, partial + (int64_t)kRowTLo * kStatBlocks);
  block_sum_dd(qh, ql, partial + (int64_t)kRowT2 * kStatBlocks, partial + (int64_t)kRowT2Lo * kStatBlocks);
}

__global__ void __launch_bounds__(kStatThreads) k_stats_pass2(const double* __restrict__ vec,
                                                              const int32_t* __restrict__ state, int64_t n,
                                                              const double* __restrict__ sums1,
                                                              double* __restrict__ partial) {
  double acc[kStatPass2] = {0};
  const double cnt = sums1[0];
  double a[6];
#pragma unroll
  for (int i = 0; i < 6; i++) a[i] = cnt > 0 ? sums1[1 + i] / cnt : 0.0;
  for (int64_t j = (int64_t)blockIdx.x * kStatThreads + threadIdx.x; j < n; j += (int64_t)gridDim.x * kStatThreads) {
    const int32_t st = state[j];
    double d[6];
#pragma unroll
    for (int i = 0; i < 6; i++) d[i] = vec[i * n + j];
    if (st != 1) continue;
#pragma unroll
    for (int i = 0; i < 6; i++) d[i] = d[i] - a[i];
    int k = 0;
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
      for (int m = i; m < 6; m++) acc[k++] += d[i] * d[m];
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const double d2 = d[i] * d[i];
      acc[21 + i] += d2 * d[i];
      acc[27 + i] += d2 * d2;
    }
  }
  block_sum<kStatPass2>(acc, partial);
}

// out[k] = the sum of row k of partial, one warp per value; with_t: rows kRowT and kRowT2 have low parts.
__global__ void __launch_bounds__(1024) k_stats_reduce(const double* __restrict__ partial, int nv, int with_t,
                                                       double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < nv; k += 32) {
    const double* row = partial + (int64_t)k * kStatBlocks;
    if (with_t && (k == kRowT || k == kRowT2)) {
      const double* low = partial + (int64_t)(k == kRowT ? kRowTLo : kRowT2Lo) * kStatBlocks;
      double h = 0, l = 0;
      for (int b = lane; b < kStatBlocks; b += 32) {
        add_dd(h, l, row[b]);
        l += low[b];
      }
      warp_sum_dd(h, l);
      if (lane == 0) out[k] = isfinite(h) ? h + l : h;  // l is NaN once h overflows
      continue;
    }
    double s = 0;
#pragma unroll 4
    for (int b = lane; b < kStatBlocks; b += 32) s += row[b];
    s = warp_sum(s);
    if (lane == 0) out[k] = s;
  }
}

}  // namespace

cudaError_t launch_bunch_sums(const double* vec, const double* t, const int32_t* state, int64_t n, double* partial,
                              double* sums, cudaStream_t stream) {
  k_stats_pass1<<<kStatBlocks, kStatThreads, 0, stream>>>(vec, t, state, n, partial);
  k_stats_reduce<<<1, 1024, 0, stream>>>(partial, kStatPass1, 1, sums);
  k_stats_pass2<<<kStatBlocks, kStatThreads, 0, stream>>>(vec, state, n, sums, partial);
  k_stats_reduce<<<1, 1024, 0, stream>>>(partial, kStatPass2, 0, sums + kStatPass1);
  return cudaGetLastError();
}

}  // namespace bmadgpu
