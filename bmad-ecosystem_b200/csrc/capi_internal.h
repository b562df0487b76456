// capi_internal.h -- context and lattice objects shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../include/bmadgpu.h"
#include "lattice.h"
#include "track.cuh"

struct bmadgpu_ctx;

namespace bmadgpu {
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);
Globals make_globals(const bmadgpu_param& p);
// Reads and clears the context's device error flag (synchronises the context stream).
int check_err_flag(bmadgpu_ctx* c);
// Enqueues n_turns of tracking of a device-resident bunch on the context stream with the
// context's tuning (chunks of turns_per_launch, live-list compaction between them); d_moments,
// if not NULL, receives the per-turn sums [n_turns][28]. ref: in the reference's element order (TrackArgs::ref).
int track_device(bmadgpu_ctx* c, const bmadgpu_lattice* lat, const bmadgpu_bunch* b, int32_t ix_start,
                 int32_t ix_end, int32_t turn0, int32_t n_turns, double* d_moments, bool ref = false);
// Frequency-map tunes of n particles from their record hist [6][n_turn][n] (fma.cu): fstate[i]
// = 1 where state[i] is not alive, else rec_state[i]; tunes [n][6] where fstate is 0.
cudaError_t fma_launch_tunes(const double* hist, int64_t n, int32_t n_turn, int32_t N, const int32_t* state,
                             const int32_t* rec_state, int32_t* fstate, int32_t flip_a, int32_t flip_b, double* tunes,
                             int sm_count, cudaStream_t s);
}  // namespace bmadgpu

#define CUDA_TRY(call)                                            \
  do {                                                            \
    cudaError_t e_ = (call);                                      \
    if (e_ != cudaSuccess) return bmadgpu::cuda_fail(e_, #call);  \
  } while (0)

struct bmadgpu_ctx {
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;
  int32_t* d_err = nullptr;
  int64_t* d_nwork = nullptr;     // [2] live-list lengths
  int32_t* d_live[2] = {nullptr, nullptr};
  int64_t live_cap = 0;
  // staging for the host-pointer API
  int64_t cap = 0;
  double* d_vec = nullptr;
  double* d_beta = nullptr;
  double* d_t = nullptr;
  double* d_mom = nullptr;
  int64_t mom_cap = 0;
  int32_t* d_i32 = nullptr;       // state, ix_ele, ix_turn, location: 4 * cap
  bmadgpu_tuning tuning;
  int64_t launches = 0;           // kernel launches enqueued
  // scratch of the calls that need some for their own duration (Workspace), kept up to kKeptWork bytes
  void* d_work = nullptr;
  size_t work_cap = 0;
  int64_t scratch_limit = 0;      // bmadgpu_selftest_scratch_limit
  // autotuner trial copies
  int64_t tune_cap = 0;
  double* d_tvec = nullptr;
  double* d_tbeta = nullptr;
  int32_t* d_tstate = nullptr;
};

// Device scratch for one call on a context: the context's own block, grown as needed and kept for the
// next call (allocating and freeing 16 bytes a particle took longer than the statistics it served), or, above
// kKeptWork, a block freed with this object. A context is one host thread's and its work is ordered by its
// stream; every user waits for its stream before it returns.
constexpr size_t kKeptWork = (size_t)128 << 20;
struct Workspace {
  bmadgpu_ctx* c;
  void* ptr = nullptr;
  bool own = false;
  explicit Workspace(bmadgpu_ctx* ctx) : c(ctx) {}
  Workspace(const Workspace&) = delete;
  Workspace& operator=(const Workspace&) = delete;
  ~Workspace() {
    if (own) cudaFree(ptr);
  }
  // False if there is no memory for it; a caller that can do with less may ask again.
  bool get(size_t bytes) {
    if (c->scratch_limit > 0 && bytes > (size_t)c->scratch_limit) return false;
    if (bytes > kKeptWork) {
      own = cudaMalloc(&ptr, bytes) == cudaSuccess;
      if (!own) cudaGetLastError();  // handled: not the next launch's error
      return own;
    }
    if (bytes > c->work_cap) {
      cudaFree(c->d_work);
      c->d_work = nullptr;
      c->work_cap = 0;
      if (cudaMalloc(&c->d_work, bytes) != cudaSuccess) {
        cudaGetLastError();
        c->d_work = nullptr;
        return false;
      }
      c->work_cap = bytes;
    }
    ptr = c->d_work;
    return true;
  }
};

struct bmadgpu_lattice {
  int device = 0;
  bmadgpu::PackedLattice pk;
  uint8_t* d_table = nullptr;
  double* d_prefix = nullptr;
  bmadgpu::Globals G;
  bmadgpu_param param;
  std::vector<bmadgpu_element> eles;  // the element records as given (attribute look-ups)
};

