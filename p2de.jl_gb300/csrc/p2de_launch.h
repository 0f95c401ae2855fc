// Per-N1D launchers of the stage kernels (instantiated in p2de_stage_n<N1D>.cu).
#pragma once

#include <cuda_runtime.h>

#include "p2de_args.h"

namespace p2de {

struct StageGeometry {
  int elems_per_block;      // default
  int elems_per_block_max;  // largest allowed (shared-memory limit)
  int threads;
  size_t smem_a;
  size_t smem_b;
  int fbar_per_elem;  // doubles of subcell flux data per element
  int nsf;            // subcell faces per direction (Nq + N1D)
  int elems_per_block_gauss;      // the same two for GaussCollocation's kernel A
  int elems_per_block_max_gauss;
  int elems_per_block_flux;  // and for kernel A in flux form
  int elems_per_block_max_flux;
};

// Default threads per block of kernel A in flux form. Its longest phase, the lines, fills 64
// threads at the default elements per block, and 128 leave half the block at that phase's
// barrier (DMR 480x120 N=3: 776 us a stage with 128 threads, 656 with 64; KH 192x192 N=5:
// 1659 and 1376). With few blocks per SM the shorter phases count, which 128 threads halve
// (Riemann 64x64 N=4, 4.5 blocks an SM: 192 us with 128, 213 with 64).
inline int flux_threads(int K, int epb) { return (K + epb - 1) / epb < 10 * 152 ? 128 : 64; }

template <int N1D>
cudaError_t stage_prepare(StageGeometry* geo);
template <int N1D>
cudaError_t launch_stage_a(const StageArgs& a, bool mixed, cudaStream_t st);
template <int N1D>
cudaError_t launch_stage_b(const StageArgs& a, cudaStream_t st);
template <int N1D>
cudaError_t launch_gauss_proj(const StageArgs& a, cudaStream_t st);
template <int N1D>
cudaError_t launch_es_interface(const StageArgs& a, cudaStream_t st);

// Per-element geometry factors (geom_factor) for K elements: out has 16 doubles per element.
cudaError_t launch_geom_table(const double* geom, int K, double* out, cudaStream_t st);

}  // namespace p2de
