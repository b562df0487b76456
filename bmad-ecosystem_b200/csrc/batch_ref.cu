// batch_ref.cu -- the instantiations of k_batch_track with the reference's element order inline
// (batch_kernel.cuh, REF), for lattices without forms in fastmaps.cuh for many of their elements. The correctly
// rounded build tracks everything in that order and has none.

#include <cuda_runtime.h>

#include "batch.cuh"
#include "batch_kernel.cuh"

namespace bmadgpu {

#if defined(BG_FAST_MAPS)

const void* batch_ref_kernel(int block, int minb, bool full) {
  struct Entry {
    int block, minb;
    const void* fn;
    const void* fn_lean;
  };
#define BG_BATCH_REF(B, M) \
  {B, M, (const void*)k_batch_track<B, M, false, true, true>, (const void*)k_batch_track<B, M, false, false, true>}
  static const Entry kRef[] = {BG_REF_SHAPES(BG_BATCH_REF)};
#undef BG_BATCH_REF
  for (const Entry& e : kRef)
    if (e.block == block && e.minb == minb) return full ? e.fn : e.fn_lean;
  return nullptr;
}

// This translation unit's copy of the __constant__ multipole tables.
cudaError_t batch_ref_upload_constants() {
  double cm[22][22], cf[22][22];
  build_cmulti_tables(cm, cf);
  cudaError_t e = cudaMemcpyToSymbol(c_cmulti, cm, sizeof(cm));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_cfull, cf, sizeof(cf));
}

#else

const void* batch_ref_kernel(int, int, bool) { return nullptr; }
cudaError_t batch_ref_upload_constants() { return cudaSuccess; }

#endif

}  // namespace bmadgpu
