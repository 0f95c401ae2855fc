// Batched stage kernel A with FP32 flux differencing (mixed precision).
#include "p2de_batch_kernels.cuh"

namespace p2de {

cudaError_t batch_prepare_f64();
cudaError_t batch_occupancy_a_f64(int kind, size_t smem, int* bpa);
cudaError_t launch_batch_a_f64(int kind, int mode, int grid, size_t smem, const StageArgs* solves,
                               const BatchTask* tasks, const int* ntasks, unsigned* counter, int nstage,
                               cudaStream_t st);

cudaError_t batch_prepare(bool mixed) {
  cudaError_t e = batch_prepare_f64();
  if (e != cudaSuccess || !mixed) return e;
  const struct {
    const void* f;
    size_t smem;
  } k[] = {{(const void*)k_batch_a<float, false>, kBatchSmemAMax},
           {(const void*)k_batch_a<float, true>, kBatchSmemXMax},
           {(const void*)k_batch_flux_a<float, false>, kBatchSmemFluxMax<false>},
           {(const void*)k_batch_flux_a<float, true>, kBatchSmemFluxMax<true>}};
  for (const auto& q : k) {
    e = cudaFuncSetAttribute(q.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q.smem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t batch_occupancy_a(bool mixed, int kind, size_t smem, int* bpa) {
  if (!mixed) return batch_occupancy_a_f64(kind, smem, bpa);
  const void* k[] = {(const void*)k_batch_a<float, false>, (const void*)k_batch_a<float, true>,
                     (const void*)k_batch_flux_a<float, false>, (const void*)k_batch_flux_a<float, true>};
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpa, k[kind], kBatchThreads, smem);
}

cudaError_t launch_batch_a(bool mixed, int kind, int mode, int grid, size_t smem, const StageArgs* solves,
                           const BatchTask* tasks, const int* ntasks, unsigned* counter, int nstage, cudaStream_t st) {
  if (!mixed) return launch_batch_a_f64(kind, mode, grid, smem, solves, tasks, ntasks, counter, nstage, st);
  if (kind == BATCH_EXT)
    k_batch_a<float, true><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  else if (kind == BATCH_PLAIN)
    k_batch_a<float, false><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  else if (kind == BATCH_FLUX_EXT)
    k_batch_flux_a<float, true><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  else
    k_batch_flux_a<float, false><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  return cudaGetLastError();
}

}  // namespace p2de
