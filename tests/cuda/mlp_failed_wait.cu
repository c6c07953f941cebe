// A training step whose pass reports a wait that gave up: the flags it would
// set are set by hand before the step.  The step fails, and parameters,
// moments and step count stay as they were: the next step gives what it gives
// without the failed one.  And a wait for an arrival that never comes, by itself.
// Build: nvcc -gencode arch=compute_103a,code=sm_103a -std=c++17
#include "../../ryr_hyperactivity_gb300/csrc/mlp.cu"

#include <vector>

__global__ void wait_kernel(int* gave_up) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc::saddr(&bar)) : "memory");
  __syncthreads();
  if (!tc::mbar_wait(tc::saddr(&bar), 0)) *gave_up = 1;  // nothing ever arrives
}

int main() {
  constexpr int n = 300;
  std::vector<float> p(kNPar), x(4 * n), t(3 * n), before(kNPar), after(kNPar), a(kNPar), b(kNPar);
  for (int i = 0; i < kNPar; ++i) p[i] = 0.1f * (float)((i * 7919) % 201 - 100) / 100.f;
  for (int i = 0; i < 4 * n; ++i) x[i] = (float)((i * 104729) % 1000) / 1000.f;
  for (int i = 0; i < 3 * n; ++i) t[i] = (float)((i * 1299709) % 500) / 1000.f;
  rh_mlp *u = nullptr, *w = nullptr;
  if (rh_mlp_create(n, 0, &u) || rh_mlp_create(n, 0, &w)) return 2;
  float loss = 0;
  for (rh_mlp* m : {u, w})
    if (rh_mlp_set_params(m, p.data()) || rh_mlp_train_step(m, x.data(), t.data(), n, 1e-2f, &loss))
      return 3;
  if (rh_mlp_get_params(w, before.data())) return 4;
  *w->h_err = 1;
  const int one = 1;
  if (cudaMemcpy(w->failed, &one, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) return 5;
  // another batch, so that its gradients are not those of the first step
  const int rc = rh_mlp_train_step(w, x.data() + 4, t.data() + 3, n - 1, 1e-2f, &loss);
  if (rh_mlp_get_params(w, after.data())) return 6;
  const bool kept = !memcmp(before.data(), after.data(), kNPar * sizeof(float));
  for (rh_mlp* m : {u, w})
    if (rh_mlp_train_step(m, x.data(), t.data(), n, 1e-2f, &loss)) return 7;
  if (rh_mlp_get_params(u, a.data()) || rh_mlp_get_params(w, b.data())) return 8;
  const bool same = !memcmp(a.data(), b.data(), kNPar * sizeof(float));
  const bool moved = memcmp(a.data(), before.data(), kNPar * sizeof(float)) != 0;
  printf("timeout %d kept %d same %d moved %d\n", rc == RH_ERR_TIMEOUT, kept, same, moved);
  int *flag = nullptr, gave_up = 0;
  float ms = 0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  if (cudaMalloc(&flag, sizeof(int)) != cudaSuccess || cudaMemset(flag, 0, sizeof(int)) != cudaSuccess)
    return 9;
  cudaEventRecord(e0);
  wait_kernel<<<1, 512>>>(flag);
  cudaEventRecord(e1);
  if (cudaMemcpy(&gave_up, flag, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 10;
  cudaEventElapsedTime(&ms, e0, e1);
  printf("wait gave up %d within 3 s %d (%.0f ms)\n", gave_up, ms < 3000.f, ms);
  rh_mlp_destroy(u);
  rh_mlp_destroy(w);
  return 0;
}
