// Launchers of the batched stage kernels (p2de_batch_f64.cu, p2de_batch_f32.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "p2de_args.h"

namespace p2de {

struct BatchTask;

// Instantiations of batched kernel A by member: the nodal-form stage body, plain or EXT, and
// the flux-form one (F_FLUX), plain or EXT.
enum : int { BATCH_PLAIN = 0, BATCH_EXT = 1, BATCH_FLUX = 2, BATCH_FLUX_EXT = 3, BATCH_KINDS = 4 };
inline int batch_kind(int flags) {
  return ((flags & F_FLUX) ? BATCH_FLUX : BATCH_PLAIN) + ((flags & kExtFlags) ? 1 : 0);
}

// Sets the kernels' largest shared-memory limits.
cudaError_t batch_prepare(bool mixed);
// Resident blocks per SM of kernel A of a kind at the given dynamic shared memory, and of
// kernel B (flux form or not).
cudaError_t batch_occupancy_a(bool mixed, int kind, size_t smem, int* blocks_per_sm);
cudaError_t batch_occupancy_b(bool flux, size_t smem, int* blocks_per_sm);
// Batched kernel A over a task list: a kind, full or low-only pass (mode).
cudaError_t launch_batch_a(bool mixed, int kind, int mode, int grid, size_t smem, const StageArgs* solves,
                           const BatchTask* tasks, const int* ntasks, unsigned* counter, int nstage, cudaStream_t st);
// initialize_s_modified! of the members with a relaxed min-entropy bound (one block per slot).
cudaError_t launch_batch_phi_min(const StageArgs* solves, const uint8_t* active, int nslots, cudaStream_t st);
cudaError_t launch_batch_b(bool flux, int grid, size_t smem, const StageArgs* solves, const BatchTask* tasks, const int* ntasks,
                           unsigned* counter, int nstage, cudaStream_t st);
cudaError_t launch_batch_begin(const StageArgs* solves, const uint8_t* active, int nslots, unsigned* counters,
                               cudaStream_t st);
int batch_elems_per_block(int n1d, bool flux);  // default
int batch_elems_per_block_max(int n1d);         // shared-memory limit of every kind
size_t batch_smem_a(int n1d, int epb, int kind);
size_t batch_smem_b(int n1d, int epb);

}  // namespace p2de
