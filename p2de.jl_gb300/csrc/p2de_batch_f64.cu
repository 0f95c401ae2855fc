// Batched stage kernels, FP64 flux differencing; kernels B and the step begin.
#define P2DE_BATCH_COMMON_KERNELS
#include "p2de_batch_kernels.cuh"

namespace p2de {

cudaError_t batch_prepare_f64() {
  const struct {
    const void* f;
    size_t smem;
  } k[] = {{(const void*)k_batch_a<double, false>, kBatchSmemAMax},
           {(const void*)k_batch_a<double, true>, kBatchSmemXMax},
           {(const void*)k_batch_flux_a<double, false>, kBatchSmemFluxMax<false>},
           {(const void*)k_batch_flux_a<double, true>, kBatchSmemFluxMax<true>},
           {(const void*)k_batch_b, kBatchSmemBMax}};
  for (const auto& q : k) {
    cudaError_t e = cudaFuncSetAttribute(q.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q.smem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t batch_occupancy_a_f64(int kind, size_t smem, int* bpa) {
  const void* k[] = {(const void*)k_batch_a<double, false>, (const void*)k_batch_a<double, true>,
                     (const void*)k_batch_flux_a<double, false>, (const void*)k_batch_flux_a<double, true>};
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpa, k[kind], kBatchThreads, smem);
}

cudaError_t batch_occupancy_b(bool flux, size_t smem, int* bpb) {
  return flux ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpb, k_batch_flux_b, kBatchThreads, 0)
              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(bpb, k_batch_b, kBatchThreads, smem);
}

cudaError_t launch_batch_a_f64(int kind, int mode, int grid, size_t smem, const StageArgs* solves,
                               const BatchTask* tasks, const int* ntasks, unsigned* counter, int nstage,
                               cudaStream_t st) {
  if (kind == BATCH_EXT)
    k_batch_a<double, true><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  else if (kind == BATCH_PLAIN)
    k_batch_a<double, false><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  else if (kind == BATCH_FLUX_EXT)
    k_batch_flux_a<double, true><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  else
    k_batch_flux_a<double, false><<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage, mode);
  return cudaGetLastError();
}

cudaError_t launch_batch_phi_min(const StageArgs* solves, const uint8_t* active, int nslots, cudaStream_t st) {
  k_batch_phi_min<<<nslots > 0 ? nslots : 1, 1024, 0, st>>>(solves, active, nslots);
  return cudaGetLastError();
}

cudaError_t launch_batch_b(bool flux, int grid, size_t smem, const StageArgs* solves, const BatchTask* tasks,
                           const int* ntasks, unsigned* counter, int nstage, cudaStream_t st) {
  if (flux)
    k_batch_flux_b<<<grid, kBatchThreads, 0, st>>>(solves, tasks, ntasks, counter, nstage);
  else
    k_batch_b<<<grid, kBatchThreads, smem, st>>>(solves, tasks, ntasks, counter, nstage);
  return cudaGetLastError();
}

cudaError_t launch_batch_begin(const StageArgs* solves, const uint8_t* active, int nslots, unsigned* counters,
                               cudaStream_t st) {
  int grid = (nslots + 127) / 128;
  k_batch_begin<<<grid > 0 ? grid : 1, 128, 0, st>>>(solves, active, nslots, counters);
  return cudaGetLastError();
}

template <int N1D>
static size_t smem_a_of(int epb, int kind) {
  switch (kind) {
    case BATCH_PLAIN: return Cfg<N1D>::smem_a(epb);
    case BATCH_EXT: return Cfg<N1D>::smem_x(epb);
    case BATCH_FLUX: return FluxCfg<N1D>::template smem<false, true>(epb);
    default: return FluxCfg<N1D>::template smem<true>(epb);
  }
}

int batch_elems_per_block(int n1d, bool flux) {
  switch (n1d) {
    case 2: return flux ? FluxCfg<2>::E_BATCH : Cfg<2>::E;
    case 3: return flux ? FluxCfg<3>::E_BATCH : Cfg<3>::E;
    case 4: return flux ? FluxCfg<4>::E_BATCH : Cfg<4>::E;
    case 5: return flux ? FluxCfg<5>::E_BATCH : Cfg<5>::E;
    case 6: return flux ? FluxCfg<6>::E_BATCH : Cfg<6>::E;
  }
  return 0;
}

int batch_elems_per_block_max(int n1d) {
  switch (n1d) {
    case 2: return cmin(Cfg<2>::E_MAX, FluxCfg<2>::E_SPLIT_MAX);
    case 3: return cmin(Cfg<3>::E_MAX, FluxCfg<3>::E_SPLIT_MAX);
    case 4: return cmin(Cfg<4>::E_MAX, FluxCfg<4>::E_SPLIT_MAX);
    case 5: return cmin(Cfg<5>::E_MAX, FluxCfg<5>::E_SPLIT_MAX);
    case 6: return cmin(Cfg<6>::E_MAX, FluxCfg<6>::E_SPLIT_MAX);
  }
  return 0;
}

size_t batch_smem_a(int n1d, int epb, int kind) {
  switch (n1d) {
    case 2: return smem_a_of<2>(epb, kind);
    case 3: return smem_a_of<3>(epb, kind);
    case 4: return smem_a_of<4>(epb, kind);
    case 5: return smem_a_of<5>(epb, kind);
    case 6: return smem_a_of<6>(epb, kind);
  }
  return 0;
}

size_t batch_smem_b(int n1d, int epb) {
  switch (n1d) {
    case 2: return Cfg<2>::smem_b(epb);
    case 3: return Cfg<3>::smem_b(epb);
    case 4: return Cfg<4>::smem_b(epb);
    case 5: return Cfg<5>::smem_b(epb);
    case 6: return Cfg<6>::smem_b(epb);
  }
  return 0;
}

}  // namespace p2de
