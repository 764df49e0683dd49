// jne_accum_digits.cu -- launches of the FP64 accumulation in exact digits
// (jne_accum_digits.cuh) for the engine's own increments, dims 1..6; the larger
// dims are compiled in jne_accum_digits_hi.cu (translation units built in
// parallel).  Explicit increments, whose range and precision are the caller's,
// keep the kernel of jne_accum_f64.cu.
#include "jne_accum_digits.cuh"

cudaError_t jne_launch_accum_digits(const jne_accum_args& a, const jne_finalize_args* fin, int sms, cudaStream_t st) {
  if (a.n_runs <= 0) return cudaSuccess;
  if (a.ext || !a.next_run) return cudaErrorInvalidValue;
  jne_finalize_args f{};  // out == nullptr: accumulation only
  if (fin) f = *fin;
  switch (a.dim) {
    case 1: return launch_digits_dim<1>(a, f, sms, st);
    case 2: return launch_digits_dim<2>(a, f, sms, st);
    case 3: return launch_digits_dim<3>(a, f, sms, st);
    case 4: return launch_digits_dim<4>(a, f, sms, st);
    case 5: return launch_digits_dim<5>(a, f, sms, st);
    case 6: return launch_digits_dim<6>(a, f, sms, st);
    default: return jne_launch_accum_digits_hi(a, f, sms, st);
  }
}
