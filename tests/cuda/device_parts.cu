// Device functions of the library's kernels, each run by itself on host
// arrays (loaded with ctypes by test_gpu_device_parts.py).
// Build: nvcc -gencode arch=compute_103a,code=sm_103a -std=c++17 -shared
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "../../ryr_hyperactivity_gb300/csrc/tile.cuh"

namespace {

using namespace rh;

// A host array on the device, copied back by get().
template <class T>
struct Dev {
  T* p = nullptr;
  size_t n;
  Dev(const T* h, size_t n_) : n(n_) {
    cudaMalloc(&p, n * sizeof(T));
    if (h) cudaMemcpy(p, h, n * sizeof(T), cudaMemcpyHostToDevice);
  }
  ~Dev() { cudaFree(p); }
  bool get(T* h) { return cudaMemcpy(h, p, n * sizeof(T), cudaMemcpyDeviceToHost) == cudaSuccess; }
};

__global__ void sums_kernel(const double* rows, int n, double* o) {
  output_sums_warp(rows, n, o, (int)threadIdx.x);
}

}  // namespace

extern "C" {

int part_row_length() { return P_COUNT; }
int part_first_statistic() { return P_STEP_END; }

// o[NOUT] from n rows of P_COUNT doubles
int part_output_sums(const double* rows, int n, double* o) {
  Dev<double> r(rows, (size_t)n * P_COUNT), d(nullptr, NOUT);
  sums_kernel<<<1, 32>>>(r.p, n, d.p);
  return d.get(o) ? NOUT : -1;
}

}  // extern "C"
