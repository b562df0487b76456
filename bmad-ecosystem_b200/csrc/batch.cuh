// batch.cuh -- kernel interface of batched tracking over many lattice variants (batch.cu), used
// by the batch entry points and the serving loop.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "table.h"

namespace bmadgpu {

constexpr uint32_t kMaxStageBytes = 200 * 1024;  // largest table staged in shared memory

// Per-variant descriptor in device memory (one lattice + its particles).
struct BatchVar {
  const uint8_t* table;       // packed element table
  const double* ref_prefix;   // [n_ele + 1] sums of delta_ref_time
  int64_t n;                  // particles of the variant
  int64_t off;                // index of its first particle in the batch-wide arrays
  uint32_t table_bytes, hdr_bytes, ap_bytes, n_ele;
  int32_t turn0;              // turn number of call-relative turn 0
  int32_t n_turns;            // turns of the current call for this variant
  Globals G;
  // Frequency-map job (serving): after every turn the normalised coordinates of each surviving
  // particle go to rec [6][rec_turns][n]; nullptr for every other variant.
  double* rec;
  const double* rec_par;      // norm [36] (row-major), closed orbit [6], z_limit (0: no z cut)
  int32_t* rec_state;         // [n] 0 recording, 2 stopped outside the RF bucket; [n, 2n) its turn
  int32_t rec_turn0;          // turn number of the job's first turn
  int32_t rec_turns;          // the job's turn count
};

// Arguments of one launch of k_batch_track: call-relative turns [turn_off, turn_off + n_turns),
// clipped per variant to its n_turns.
struct BatchArgs {
  const BatchVar* vars;
  int32_t n_var;
  int32_t tile;               // particles per work item (threads per CTA x particles per thread)
  double* vec;                // variant v: [6][n_v] block at vec + 6 * off_v
  double* beta;
  double* t;
  int32_t* state;
  int32_t* ix_ele;
  int32_t* ix_turn;
  int32_t* location;
  int32_t turn_off, n_turns;
  const int64_t* tile_prefix;        // [n_var + 1]: first work item of each variant
  const int32_t* live_in;            // variant v's live list at live_in + off_v; nullptr: 0 .. n_v-1
  const unsigned long long* n_in;    // [n_var] live-list lengths (unused with live_in == nullptr)
  int32_t* live_out;                 // nullptr: no compaction after this launch
  unsigned long long* n_out;         // [n_var] lengths of the compacted lists
  unsigned long long* queue;         // work-item counter, zero at launch
  int32_t* err_flag;                 // bit 0: table staging wait timed out
  uint32_t smem_bytes;               // dynamic shared memory for staging (0: read tables from global). To
                                     // batch_launch_track: what the launch's tables need (default build)
  int32_t rare;                      // some variant's table has extra blocks / pitched offsets
  int32_t ref;                       // variants that track in the reference's order (Globals::hi_hot_pz = 0):
                                     // 0 none, 1 some (tile_prefix and queue hold a second plan, for them),
                                     // 2 all
  int32_t plan_stride;               // from tile_prefix to the second plan's
};

struct BatchLaunch {
  int block = 128;
  int ctas_per_sm = 0;        // register budget selector, as LaunchCfg::ctas_per_sm
  int particles_per_thread = 1;
  int ref_ctas = -1;          // the same for the kernels in the reference's order; -1: as ctas_per_sm
};

// Which instantiation a launch takes: the forms of fastmaps.cuh, or with the reference's element forms inline
// for every element form (full) or for tables without rare ones (lean, TableInfo::rare).
enum BatchForm : int { kBatchForms = 0, kBatchFull = 1, kBatchLean = 2 };

// Kernels + grids of a launch shape (resolved once, outside stream capture).
struct BatchKernel {
  int block = 0, ppt = 1;
  const void* fn[3][2] = {};     // [BatchForm][with the frequency-map record path]
  int grid[3][2] = {};
  uint32_t smem[3][2] = {};      // shared memory for staging: the room for it (default build), else what is taken
};

cudaError_t batch_upload_constants();
// The other translation units' copies of the tables (those of the reference's order filled by batch_resolve,
// so that a context loads them only when it wants them), and their instantiations of a shape: with the record
// path (full: every element form, else the lean one), in the reference's order (default build; shapes of
// BG_REF_SHAPES, else null), and with both.
cudaError_t batch_rec_upload_constants();
cudaError_t batch_ref_upload_constants();
cudaError_t batch_ref_rec_upload_constants();
const void* batch_rec_kernel(int block, int minb, bool full = true);
const void* batch_ref_kernel(int block, int minb, bool full);
const void* batch_ref_rec_kernel(int block, int minb, bool full);
// ref (as BatchArgs::ref): which sorts of lattice; a kernel that is not wanted is not loaded, since its stack
// would widen every kernel's local memory (a served burst of small jobs took 4 % longer).
// smem_bytes: shared memory for staging, as much as the largest table that may be staged; 0: none. The default
// build stages lattices in the reference's order alone, tables up to what leaves the resident CTAs unchanged.
cudaError_t batch_resolve(const BatchLaunch& cfg, int ref, uint32_t smem_bytes, int sm_count, BatchKernel* out);
// record: use the instantiation with the frequency-map record path (rounds with an FMA job). *launches: kernels
// launched.
cudaError_t batch_launch_track(const BatchKernel& k, const BatchArgs& a, cudaStream_t stream, bool record,
                               int64_t* launches);
// Work plan for a launch: tile_prefix from the live counts (or the variants' sizes when
// identity is set), restricted to variants with turns left after turn_off; zeroes the queue
// counter and the next launch's counts (n_zero, nullable). With variants of both sorts (ref 1) two plans: of those
// in the forms of fastmaps.cuh to tile_prefix and queue[0], of those in the reference's order to
// tile_prefix + plan_stride and queue[1].
cudaError_t batch_launch_plan(const BatchVar* vars, int32_t n_var, int32_t tile, int32_t turn_off, bool identity,
                              const unsigned long long* n_in, int64_t* tile_prefix, unsigned long long* queue,
                              unsigned long long* n_zero, int ref, int32_t plan_stride, cudaStream_t stream,
                              int64_t* launches);
// Sets turn0 and n_turns of every variant (the batch entry point's per-call values).
cudaError_t batch_launch_set_turns(BatchVar* vars, int32_t n_var, int32_t turn0, int32_t n_turns,
                                   cudaStream_t stream);

// A job's first live list: list[i] = i for i < n, *count = n.
cudaError_t batch_launch_init_list(int32_t* list, int64_t n, unsigned long long* count, cudaStream_t stream);

}  // namespace bmadgpu
