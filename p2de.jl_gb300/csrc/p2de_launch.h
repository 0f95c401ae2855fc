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

// Launch shape of kernel A in flux form: the layout of its lines (FluxLine: one thread a line,
// or split), and the default elements and threads per block.
//  * Split below 64k nodes (110k from N = 4 on, whose lines are longer): there an SM has so few
//    warps that a line's chain is the stage's duration, and small blocks spread the elements
//    evenly over the SMs. Measured, one thread a line against split, us a stage: KH 32x32 N=3
//    37.4 and 26.9, 5x5 N=3 33.2 and 18.0, 16x16 N=2 26.7 and 17.0, 32x32 N=5 74.7 and 59.6,
//    Riemann 64x64 N=4 with the intended bounds 206 and 157; KH 64x64 N=3 57.9 and 61.7, DMR
//    480x120 N=3 611 and 645. The EXT modes (their time is in the bounds) keep the lines.
//  * 64 threads otherwise: the lines fill them at the default elements per block, and 128 leave
//    half the block at that phase's barrier (DMR 480x120 N=3 776 and 656 us, KH 192x192 N=5
//    1659 and 1376); 128 where a grid is under ten blocks an SM and the shorter phases count,
//    and at N = 2, whose 10 elements fill 128 with nodes (240x120: 220 and 190 us). With FP32
//    pairs (acc64) the node phases weigh more: N = 5 takes 6 elements and 128 threads (192x192:
//    841 us against 941 with 5 and 64), N = 4 takes 5 elements (460 against 520 with 6).
struct FluxShape {
  bool split;
  int epb, threads;
};
// sms: multiprocessors of the device.
inline FluxShape flux_shape(int n1d, int K, int epb_lines, bool ext, bool acc64, int sms) {
  const int64_t nodes = (int64_t)K * n1d * n1d;
  if (!ext && nodes < (n1d >= 5 ? 110000 : 65536))
    return {true, n1d == 2 ? 8 : n1d == 3 || n1d == 5 ? 3 : 2, 128};
  if (acc64 && n1d >= 5) epb_lines = n1d == 5 ? 5 : 6;
  const bool wide = n1d == 3 || (acc64 && n1d == 6) || (K + epb_lines - 1) / epb_lines < 10 * sms;
  return {false, epb_lines, wide ? 128 : 64};
}

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
