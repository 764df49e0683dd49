// jne_finalize.cu -- the finalize kernel: one thread per run turns the run's
// moment record into its eigenvalues (jne_finalize_run.cuh; replaces
// johansen_statistics.rs:24-47).  Used by multi-model requests (one accumulation,
// then every model of every run in one launch) and by explicit increments in
// FP64; the other kernels finalize their own runs.
#include "jne_finalize_run.cuh"

namespace {

// Blocks of two warps, and all models in one grid, so that only the launch's own
// tail leaves SMs idle.  As many blocks per SM as registers allow: the local arrays
// then miss L1, but the warps hide it (five models of 40,000 runs at k = 12, 13: 4.0
// ms with 18 blocks per SM, 4.4 with 8, 5.2 with 4, 6.5 with 2).
constexpr int kFinThreads = 64;

struct FinalizeList {
  jne_finalize_args f[5];
};

__global__ void __launch_bounds__(kFinThreads) k_finalize(const __grid_constant__ FinalizeList list) {
  const jne_finalize_args& f = list.f[blockIdx.y];
  const int run = blockIdx.x * kFinThreads + threadIdx.x;
  if (run < f.n_runs) jne_fin::finalize_run<true>(f, run);
}

}  // namespace

cudaError_t jne_launch_finalize(const jne_finalize_args* f, int n, cudaStream_t st) {
  if (n < 1 || n > 5) return cudaErrorInvalidValue;
  if (f[0].n_runs <= 0) return cudaSuccess;
  FinalizeList list{};
  for (int i = 0; i < n; i++) list.f[i] = f[i];
  const dim3 grid((f[0].n_runs + kFinThreads - 1) / kFinThreads, n);
  k_finalize<<<grid, kFinThreads, 0, st>>>(list);
  return cudaGetLastError();
}
