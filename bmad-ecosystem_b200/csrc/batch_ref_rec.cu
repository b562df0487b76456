// batch_ref_rec.cu -- the instantiations of batch_ref.cu with the frequency-map record path, a file of
// their own so that the two compile in parallel.

#include <cuda_runtime.h>

#include "batch.cuh"
#include "batch_kernel.cuh"

namespace bmadgpu {

#if defined(BG_FAST_MAPS)

const void* batch_ref_rec_kernel(int block, int minb, bool full) {
  struct Entry {
    int block, minb;
    const void* fn;
    const void* fn_lean;
  };
#define BG_BATCH_REF(B, M) \
  {B, M, (const void*)k_batch_track<B, M, true, true, true>, (const void*)k_batch_track<B, M, true, false, true>}
  static const Entry kRef[] = {BG_REF_SHAPES(BG_BATCH_REF)};
#undef BG_BATCH_REF
  for (const Entry& e : kRef)
    if (e.block == block && e.minb == minb) return full ? e.fn : e.fn_lean;
  return nullptr;
}

// This translation unit's copy of the __constant__ multipole tables.
cudaError_t batch_ref_rec_upload_constants() {
  double cm[22][22], cf[22][22];
  build_cmulti_tables(cm, cf);
  cudaError_t e = cudaMemcpyToSymbol(c_cmulti, cm, sizeof(cm));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_cfull, cf, sizeof(cf));
}

#else

const void* batch_ref_rec_kernel(int, int, bool) { return nullptr; }
cudaError_t batch_ref_rec_upload_constants() { return cudaSuccess; }

#endif

}  // namespace bmadgpu
