// The kernels' point arithmetic (p2de_arith.cuh) over arrays, for its tests (in
// libp2de_probe.so, not part of the solver library). Returns 0 on success, 1 on a bad argument,
// 3 on a CUDA error.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../p2de_arith.cuh"
#include "../p2de_tables.h"

namespace {

enum : int { OP_RCP = 0, OP_SQRT = 1, OP_DIV = 2, OP_LOG = 3, OP_LOG_HALF = 4, OP_EXP = 5, OP_POW = 6, OP_COUNT = 7 };

__global__ void k_arith(int op, int64_t n, const double* a, const double* b, double* out, const p2de::LineOps* tab) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  switch (op) {
    case OP_RCP: out[i] = p2de::rcp(a[i]); break;
    case OP_SQRT: out[i] = p2de::sqrt_rn(a[i]); break;
    case OP_DIV: out[i] = p2de::div_rn(a[i], b[i]); break;
    case OP_LOG: out[i] = p2de::log_fast(a[i], *tab); break;
    case OP_LOG_HALF: out[i] = p2de::log_fast<true>(a[i], *tab); break;
    case OP_EXP: out[i] = p2de::exp_fast(a[i], *tab); break;
    case OP_POW: out[i] = p2de::pow_fast(a[i], b[i], *tab); break;
  }
}

}  // namespace

// out[i] = op(a[i], b[i]) for n host arrays' elements
extern "C" int p2de_probe_arith(int device, int32_t op, int64_t n, const double* a, const double* b, double* out) {
  if (op < 0 || op >= OP_COUNT || n < 1 || n > (int64_t)1 << 30 || !a || !b || !out) return 1;
  static p2de::LineOps host;
  if (p2de::build_line_ops(1, 5e-16, &host, 0) != 0) return 1;
  if (cudaSetDevice(device) != cudaSuccess) return 3;
  const size_t bytes = sizeof(double) * (size_t)n;
  double* d[3] = {nullptr, nullptr, nullptr};
  p2de::LineOps* tab = nullptr;
  cudaError_t e = cudaMalloc(&tab, sizeof host);
  for (int i = 0; i < 3 && e == cudaSuccess; ++i) e = cudaMalloc(&d[i], bytes);
  if (e == cudaSuccess) e = cudaMemcpy(tab, &host, sizeof host, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_arith<<<(unsigned)((n + 255) / 256), 256>>>(op, n, d[0], d[1], d[2], tab);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d[2], bytes, cudaMemcpyDeviceToHost);
  for (double* p : d) cudaFree(p);
  cudaFree(tab);
  return e == cudaSuccess ? 0 : 3;
}
