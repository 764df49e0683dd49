// jne_accum_digits_hi.cu -- the FP64 accumulation in exact digits, dims 7..12
// (see jne_accum_digits.cu).
#include "jne_accum_digits.cuh"

cudaError_t jne_launch_accum_digits_hi(const jne_accum_args& a, const jne_finalize_args& f, int sms, cudaStream_t st) {
  switch (a.dim) {
    case 7: return launch_digits_dim<7>(a, f, sms, st);
    case 8: return launch_digits_dim<8>(a, f, sms, st);
    case 9: return launch_digits_dim<9>(a, f, sms, st);
    case 10: return launch_digits_dim<10>(a, f, sms, st);
    case 11: return launch_digits_dim<11>(a, f, sms, st);
    case 12: return launch_digits_dim<12>(a, f, sms, st);
    default: return cudaErrorInvalidValue;
  }
}
