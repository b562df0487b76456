// batch.cu -- batched tracking of many lattice variants in one persistent launch.
//
// k_batch_track: a persistent grid (one full wave of CTAs) pulls work items from a device
// counter. An item is (variant, tile of `tile` consecutive entries of the variant's live list);
// items of variant v are numbered tile_prefix[v] .. tile_prefix[v+1]-1. A CTA that moves to a
// new variant takes up that variant's element table: the element forms of the default build read it from
// global memory through L1; the correctly rounded build, and lattices in the reference's order, re-stage it
// into shared memory with a bulk copy (mbarrier completion, bounded wait, the phase bit flipping on every
// use). Each thread tracks
// `ppt` particles of the tile one after another, each through all turns of the launch, with the
// same per-particle code as k_track (particle.cuh). Survivors are appended to the variant's next
// live list with a warp ballot and one atomic per warp, so compaction needs no extra pass.
//
// k_batch_plan: one CTA; exclusive scan of the tile counts (live count / tile, rounded up) over
// the variants (want 0 or 1: of those in the forms of fastmaps.cuh or in the reference's order, each with a
// plan of its own in a launch of both), reset of the work counter and of the next launch's live counts.

#include <cuda_runtime.h>

#include <algorithm>

#include "batch.cuh"
#include "batch_kernel.cuh"
#include "particle.cuh"
#include "tma.cuh"
#include "track.cuh"

namespace bmadgpu {

namespace {

__global__ void k_batch_plan(const BatchVar* __restrict__ vars, int n_var, int tile, int turn_off, int identity, int want,
                             const unsigned long long* __restrict__ n_in, int64_t* __restrict__ tile_prefix,
                             unsigned long long* __restrict__ queue, unsigned long long* __restrict__ n_zero) {
  __shared__ long long warp_sums[32];
  __shared__ long long carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  if (threadIdx.x == 0) {
    carry = 0;
    *queue = 0;
  }
  __syncthreads();
  for (int base = 0; base < n_var; base += blockDim.x) {
    const int v = base + threadIdx.x;
    long long tiles = 0;
    if (v < n_var) {
      const long long cnt = identity ? (long long)vars[v].n : (long long)n_in[v];
      const bool mine = want < 0 || (vars[v].G.hi_hot_pz == 0) == (want != 0);
      if (mine && vars[v].n_turns > turn_off && cnt > 0) tiles = (cnt + tile - 1) / tile;
      if (n_zero) n_zero[v] = 0;
    }
    long long x = tiles;  // inclusive scan within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      long long s = lane < n_warps ? warp_sums[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      warp_sums[lane] = s;
    }
    __syncthreads();
    const long long excl = carry + (warp > 0 ? warp_sums[warp - 1] : 0) + x - tiles;
    if (v < n_var) tile_prefix[v] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + tiles;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile_prefix[n_var] = carry;
}

__global__ void k_batch_set_turns(BatchVar* vars, int n_var, int turn0, int n_turns) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n_var; v += gridDim.x * blockDim.x) {
    vars[v].turn0 = turn0;
    vars[v].n_turns = n_turns;
  }
}

__global__ void k_batch_init_list(int32_t* __restrict__ list, int64_t n, unsigned long long* __restrict__ count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    list[i] = (int32_t)i;
  if (blockIdx.x == 0 && threadIdx.x == 0) *count = (unsigned long long)n;
}

struct Variant {
  int block, minb;
  const void* fn;
  const void* fn_lean;
};
#if defined(BG_FAST_MAPS)
#define BG_BATCH_VARIANT(B, M) {B, M, (const void*)k_batch_track<B, M, false, true>, nullptr}
#else
#define BG_BATCH_VARIANT(B, M) \
  {B, M, (const void*)k_batch_track<B, M, false, true>, (const void*)k_batch_track<B, M, false, false>}
#endif
const Variant kVariants[] = {
    BG_BATCH_VARIANT(64, 4),  BG_BATCH_VARIANT(64, 8),  BG_BATCH_VARIANT(64, 12), BG_BATCH_VARIANT(128, 3),
    BG_BATCH_VARIANT(128, 4), BG_BATCH_VARIANT(128, 5), BG_BATCH_VARIANT(128, 6), BG_BATCH_VARIANT(256, 1),
    BG_BATCH_VARIANT(256, 2), BG_BATCH_VARIANT(256, 3), BG_BATCH_VARIANT(512, 1),
};
#undef BG_BATCH_VARIANT
#if defined(BG_FAST_MAPS)
#define BG_SHAPE(B, M) {B, M, nullptr, nullptr}
const Variant kRefShapes[] = {BG_REF_SHAPES(BG_SHAPE)};
#undef BG_SHAPE
#endif

// Same register-budget selection as launch_track: the largest minimum CTA count not above ctas (0: the most
// registers per thread), else the one with the most registers.
template <int N>
const Variant* pick(const Variant (&list)[N], int block, int ctas) {
  const Variant* v = nullptr;
  for (const Variant& k : list) {
    if (k.block != block) continue;
    if (ctas > 0 && k.minb > ctas) continue;
    if (!v || (ctas > 0 ? k.minb > v->minb : k.minb < v->minb)) v = &k;
  }
  if (!v)
    for (const Variant& k : list)
      if (k.block == block && (!v || k.minb < v->minb)) v = &k;
  return v;
}

}  // namespace

// The multipole coefficient tables are __constant__ arrays of each translation unit; this one
// fills the copy the batch kernel reads.
cudaError_t batch_upload_constants() {
  double cm[22][22], cf[22][22];
  build_cmulti_tables(cm, cf);
  cudaError_t e = cudaMemcpyToSymbol(c_cmulti, cm, sizeof(cm));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_cfull, cf, sizeof(cf));
}

cudaError_t batch_resolve(const BatchLaunch& cfg, int ref, uint32_t smem_bytes, int sm_count, BatchKernel* out) {
  const Variant* v = pick(kVariants, cfg.block, cfg.ctas_per_sm);
  if (!v || cfg.particles_per_thread < 1) return cudaErrorInvalidValue;
  *out = BatchKernel();
  const void* fn[3][2];
#if defined(BG_FAST_MAPS)
  const Variant* m = pick(kRefShapes, cfg.block, cfg.ref_ctas < 0 ? cfg.ctas_per_sm : cfg.ref_ctas);
  if (!m) return cudaErrorInvalidValue;
  if (ref > 0) {
    cudaError_t err = batch_ref_upload_constants();
    if (err != cudaSuccess) return err;
    if ((err = batch_ref_rec_upload_constants()) != cudaSuccess) return err;
  }
  fn[kBatchForms][0] = v->fn;
  fn[kBatchForms][1] = batch_rec_kernel(v->block, v->minb);
  for (int form : {kBatchFull, kBatchLean}) {
    fn[form][0] = batch_ref_kernel(m->block, m->minb, form == kBatchFull);
    fn[form][1] = batch_ref_rec_kernel(m->block, m->minb, form == kBatchFull);
  }
  const int first = ref < 2 ? kBatchForms : kBatchFull, last = ref > 0 ? kBatchLean : kBatchForms;
#else
  for (int form : {kBatchFull, kBatchLean}) {
    fn[form][0] = form == kBatchFull ? v->fn : v->fn_lean;
    fn[form][1] = batch_rec_kernel(v->block, v->minb, form == kBatchFull);
  }
  (void)ref;
  const int first = kBatchFull, last = kBatchLean;
#endif
  for (int form = first; form <= last; form++)
    for (int rec = 0; rec < 2; rec++) {
      const void* f = fn[form][rec];
      if (!f) return cudaErrorInvalidValue;
      uint32_t smem = form == kBatchForms ? 0 : smem_bytes;
      cudaError_t err = cudaSuccess;
      // the same limit from every caller: servers and batches share these kernels
      if (smem) err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxStageBytes);
      if (err != cudaSuccess) return err;
      int per_sm = 0;
#if defined(BG_FAST_MAPS)
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, cfg.block, 0);
      if (err != cudaSuccess) return err;
      if (smem) {  // the most that leaves the resident CTAs as they are
        size_t room = 0;
        err = cudaOccupancyAvailableDynamicSMemPerBlock(&room, f, std::max(per_sm, 1), cfg.block);
        if (err != cudaSuccess) return err;
        smem = (uint32_t)std::min<size_t>(kMaxStageBytes, room);
      }
#else
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, cfg.block, smem);
      if (err != cudaSuccess) return err;
#endif
      out->fn[form][rec] = f;
      out->grid[form][rec] = sm_count * (per_sm < 1 ? 1 : per_sm);
      out->smem[form][rec] = smem;
    }
  out->block = cfg.block;
  out->ppt = cfg.particles_per_thread;
  return cudaSuccess;
}

cudaError_t batch_launch_track(const BatchKernel& k, const BatchArgs& args_in, cudaStream_t stream, bool record,
                               int64_t* launches) {
  BatchArgs a = args_in;
  int ppt = k.ppt;
  void* args[] = {(void*)&a, (void*)&ppt};
  const int inl = a.rare ? kBatchFull : kBatchLean;
#if defined(BG_FAST_MAPS)
  const int forms[2] = {a.ref < 2 ? (int)kBatchForms : -1, a.ref > 0 ? inl : -1};
#else
  a.ref = 0;
  const int forms[2] = {inl, -1};
#endif
  for (int form : forms) {
    if (form < 0) continue;
    if (!k.fn[form][record]) return cudaErrorInvalidValue;  // not resolved
#if defined(BG_FAST_MAPS)
    // shared memory for a table that does not fit would only take it from L1 (4096 particles of a ring with
    // thin multipoles, 64 x 8: 5.3 ms against 3.3)
    a.smem_bytes = args_in.smem_bytes <= k.smem[form][record] ? args_in.smem_bytes : 0;
#else
    a.smem_bytes = k.smem[form][record];
#endif
    if (a.ref == 1 && form != kBatchForms) {  // the second plan (batch_launch_plan)
      a.tile_prefix = args_in.tile_prefix + a.plan_stride;
      a.queue = args_in.queue + 1;
    }
    cudaError_t err = cudaLaunchKernel(k.fn[form][record], dim3((unsigned)k.grid[form][record]),
                                       dim3((unsigned)k.block), args, a.smem_bytes, stream);
    if (err != cudaSuccess) return err;
    (*launches)++;
  }
  return cudaSuccess;
}

cudaError_t batch_launch_plan(const BatchVar* vars, int32_t n_var, int32_t tile, int32_t turn_off, bool identity,
                              const unsigned long long* n_in, int64_t* tile_prefix, unsigned long long* queue,
                              unsigned long long* n_zero, int ref, int32_t plan_stride, cudaStream_t stream,
                              int64_t* launches) {
#if !defined(BG_FAST_MAPS)
  ref = 0;
#endif
  for (int want = 0; want < (ref == 1 ? 2 : 1); want++) {
    k_batch_plan<<<1, 1024, 0, stream>>>(vars, n_var, tile, turn_off, identity ? 1 : 0, ref == 1 ? want : -1, n_in,
                                         tile_prefix + (int64_t)want * plan_stride, queue + want, n_zero);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    (*launches)++;
  }
  return cudaSuccess;
}

cudaError_t batch_launch_set_turns(BatchVar* vars, int32_t n_var, int32_t turn0, int32_t n_turns,
                                   cudaStream_t stream) {
  int blocks = (n_var + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 1024) blocks = 1024;
  k_batch_set_turns<<<blocks, 256, 0, stream>>>(vars, n_var, turn0, n_turns);
  return cudaGetLastError();
}

cudaError_t batch_launch_init_list(int32_t* list, int64_t n, unsigned long long* count, cudaStream_t stream) {
  int64_t blocks = (n + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 1024) blocks = 1024;
  k_batch_init_list<<<(unsigned)blocks, 256, 0, stream>>>(list, n, count);
  return cudaGetLastError();
}

}  // namespace bmadgpu
