// jne_kernels.h -- host-side launch wrappers of the device kernels.
#pragma once
#include <cuda_runtime.h>
#include "jne_common.cuh"

// Deterministic time sums over y = (i+1)/T, i = 0..T-1: Y[p] = sum y^p, p = 0..4;
// Syy = sum (y - ybar)^2, Syy2 = sum (y - ybar) y^2, Syh = sum (y - 1/2)^2, and
// Sr2, the sum of squares of y^2 less its fit on {1, y}.
struct jne_time_sums {
  double Y[5];
  double Syy, Syy2, Syh, Sr2;
};

// The mixed kernels can pack two runs into one warp ("unit") for dims up to
// this: a request of n runs is then ceil(n / 2) units, else n.
#define JNE_PACK_MAX_DIM 4
__host__ __device__ __forceinline__ long long jne_units(int dim, long long n_runs, bool pack = true) {
  return pack && dim <= JNE_PACK_MAX_DIM ? (n_runs + 1) / 2 : n_runs;
}

// Whether the mixed single-request kernel packs when nobody chose: one run per warp
// while every run has a warp of its own (4 blocks of 4 warps per SM); packed, half the
// warps would do twice the work (608 runs: dim 2, T 1000 106 -> 77 us, dim 4 210 -> 129,
// dim 3, T 10^4 284 -> 199).  From 12 runs per SM on (a fourth warp on every scheduler) long
// paths of the smallest dims are packed too, whose two runs cost little more than one:
// time unpacked over packed at 2,000 runs, T 1000, 5000, 10^4: dim 1 0.99, 1.17, 1.24; dim 2
// 0.83, 1.01, 1.11; dim 3 0.74, 0.92, 1.03; dim 4 0.67, 0.84, 0.95.
inline bool jne_pack_by_default(int dim, int steps, long long n_runs, int sms) {
  return n_runs > ((long long)steps > 1000ll * dim * dim ? 12ll : 16ll) * sms;
}

// The same for the FP64 digits (3 blocks of 4 warps per SM).  A batch of packed pairs is
// solved in two rounds, which on short paths is most of the time until the solves fill the
// GPU: time unpacked over packed at dim 4, T 33 and 2,000, 9,728, 20,000 runs 0.61, 0.72,
// 0.84; T 400 0.73, 0.95, 1.06; T 1000 and 2,000, 3,648 runs 0.80, 0.92; dim 3, T 200 and
// 2,000, 20,000 runs 0.75, 1.03; dim 2, T 100 0.75, 1.06, T 400 and 3,040 runs 1.11; dim 1 0.98
// and more past 1,824 runs.
inline bool jne_digits_pack(int dim, int steps, long long n_runs, int sms) {
  const long long line = 3000ll * dim * (dim - 1) / steps;
  return n_runs > (line < 12 ? 12 : line > 80 ? 80 : line) * sms;
}

// Argument block of the finalize kernel.
struct jne_finalize_args {
  int model, dim, steps, n_runs;
  double lam_scale;         // eigenvalues = lam_scale x those of the records' pencil (s^2 T for B = s W)
  jne_time_sums ts;
  const double* mom;        // moment records (SoA)
  long long mom_ld;
  double* out;              // n_runs x k eigenvalues, descending
  unsigned int* status;
};

// One request of a ragged batch, as the device sees it: the accumulation and
// finalize argument blocks and the request's first index in the flattened run
// space of the batch.
struct jne_ragged_req {
  jne_accum_args acc;
  jne_finalize_args fin;
  long long first;
};

// batch_done (may be null): ceil(total / 32) zeroed counts; the launch then
// also finalizes every item
cudaError_t jne_launch_accum_mixed_ragged(const jne_ragged_req* reqs, int n_req, long long total,
                                         unsigned long long* counter, unsigned int* batch_done, int sms,
                                         cudaStream_t st);
// explicit increments (a.ext) in FP64 multiply-adds over an entry table
cudaError_t jne_launch_accum_f64(const jne_accum_args& a, const int4* ent, int nent, int sms, cudaStream_t st);
// The engine's own increments (a.ext == null): every Gram sum exact in digits
// (jne_accum_digits.cuh); needs a.next_run, finalizes with fin as the mixed form.
cudaError_t jne_launch_accum_digits(const jne_accum_args& a, const jne_finalize_args* fin, int sms, cudaStream_t st);
cudaError_t jne_launch_accum_digits_hi(const jne_accum_args& a, const jne_finalize_args& f, int sms, cudaStream_t st);
int jne_build_f64_entries(int model, int d, int4* out, int cap);
// fin (may be null) finalizes the same request's runs inside the launch.
// a.blocks_per_sm (4, or 6 for the kernels budgeted to 80 registers) and
// a.pack (< 0: one run per warp at every dim) select the kernel variant.
cudaError_t jne_launch_accum_mixed(const jne_accum_args& a, const jne_finalize_args* fin, int sms, cudaStream_t st);
// the 6-blocks-per-SM variants and the explicit-increment ones (their own translation units)
cudaError_t jne_launch_accum_mixed_b6(const jne_accum_args& a, const jne_finalize_args* fin, int sms, cudaStream_t st);
cudaError_t jne_launch_accum_mixed_ext(const jne_accum_args& a, const jne_finalize_args* fin, int sms,
                                       cudaStream_t st);
// n (1..5) finalizes over the same number of runs in one launch
cudaError_t jne_launch_finalize(const jne_finalize_args* f, int n, cudaStream_t st);
// The .dat records of n results of consecutive seeds (jne_pack.cu): out is
// 16-byte aligned and holds jne_records_bytes(seed_first, n, k) bytes.
cudaError_t jne_launch_pack_records(const double* eigs, unsigned char* out, uint32_t seed_first, long long n, int k,
                                    int sms, cudaStream_t st);
cudaError_t jne_launch_export(int dim, int steps, int n_runs, uint32_t seed_first, uint32_t key0, uint32_t key1,
                              double scale, double* out, uint32_t* words, cudaStream_t st);
