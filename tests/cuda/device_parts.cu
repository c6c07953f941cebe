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

// RyR transition counts of CRU i by the FP32 estimates and by the FP64
// comparisons; est[i]: the estimates decided them all.
__global__ void draws_kernel(int n, const double* cp, const double* cjsr, const double* mono,
                             const double* ku, const double* ku2, const double* kb, double dt,
                             const int* counts, uint32_t* est, uint32_t* e, uint32_t* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  StepCoef<double> k{};
  k.ku = ku[i];
  k.ku2 = ku2[i];
  k.kb = kb[i];
  k.dt = dt;
  k.rdt = 1.0 / dt;
  rh_stream a, b;
  rh_stream_init(&a, 7u, 3u, (uint32_t)i, 5u);
  b = a;
  const int* c = counts + 4 * i;
  uint32_t status = 0;
  est[i] = ryr_draws_estimated(&a, k, cp[i], cjsr[i], mono[i], c[0], c[1], c[2], c[3], e[2 * i],
                               e[2 * i + 1])
               ? 1u + a.draw
               : 0u;
  ryr_draws<double, 1>(&b, k, cp[i], cjsr[i], mono[i], c[0], c[1], c[2], c[3], x[2 * i],
                       x[2 * i + 1], &status);
  if (est[i] && est[i] != 1u + b.draw) est[i] = 0xffffffffu;  // another number of draws taken
}

__global__ void stencil_kernel(int n, const double* v, double kt, double kl, double* o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* w = v + 12 * i;
  const double2 r = stencil_pair(make_double2(w[0], w[1]), w[2], w[3], make_double2(w[4], w[5]),
                                 make_double2(w[6], w[7]), make_double2(w[8], w[9]),
                                 make_double2(w[10], w[11]), kt, kl);
  o[2 * i] = r.x;
  o[2 * i + 1] = r.y;
}

__global__ void serca_kernel(int n, const double* v, double sviup, double* o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  serca_leak(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3], sviup, o[2 * i], o[2 * i + 1]);
}

__global__ void divide_kernel(int n, const double* a, const double* b, double* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) q[i] = div_refined(a[i], b[i]);
}

__global__ void wait_kernel(int* gave_up) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  if (!mbar_wait(&bar, 0)) *gave_up = 1;  // nothing ever arrives
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

// `in`: cp, cjsr, mono, ku, ku2, kb (n each); `counts`: nou, ncu, nob, ncb of
// each CRU; est, e[2n], x[2n] as in draws_kernel.
int part_draws(int n, const double* in, double dt, const int* counts, uint32_t* est, uint32_t* e,
               uint32_t* x) {
  const size_t m = (size_t)n;
  Dev<double> d(in, 6 * m);
  Dev<int> c(counts, 4 * m);
  Dev<uint32_t> de(nullptr, m), d0(nullptr, 2 * m), d1(nullptr, 2 * m);
  draws_kernel<<<(n + 127) / 128, 128>>>(n, d.p, d.p + m, d.p + 2 * m, d.p + 3 * m, d.p + 4 * m,
                                         d.p + 5 * m, dt, c.p, de.p, d0.p, d1.p);
  return de.get(est) && d0.get(e) && d1.get(x) ? 0 : -1;
}

// v: of each of n z-pairs its halves, outer z neighbours, inner and outer y
// and x neighbour pairs (12 doubles); o: the pair's two sums
int part_stencil(int n, const double* v, double kt, double kl, double* o) {
  Dev<double> d(v, 12 * (size_t)n), r(nullptr, 2 * (size_t)n);
  stencil_kernel<<<(n + 127) / 128, 128>>>(n, d.p, kt, kl, r.p);
  return r.get(o) ? 0 : -1;
}

// v: c, n, pa, pb of each of n sub-voxels; o: uptake and leak of each
int part_serca_leak(int n, const double* v, double sviup, double* o) {
  Dev<double> d(v, 4 * (size_t)n), r(nullptr, 2 * (size_t)n);
  serca_kernel<<<(n + 127) / 128, 128>>>(n, d.p, sviup, r.p);
  return r.get(o) ? 0 : -1;
}

int part_divide(int n, const double* a, const double* b, double* q) {
  Dev<double> da(a, (size_t)n), db(b, (size_t)n), dq(nullptr, (size_t)n);
  divide_kernel<<<(n + 127) / 128, 128>>>(n, da.p, db.p, dq.p);
  return dq.get(q) ? 0 : -1;
}

// 1 when a wait for an arrival that never comes has given up
int part_wait_runs_out() {
  const int zero = 0;
  Dev<int> d(&zero, 1);
  wait_kernel<<<1, 32>>>(d.p);
  int h = -1;
  return d.get(&h) ? h : -1;
}

}  // extern "C"
