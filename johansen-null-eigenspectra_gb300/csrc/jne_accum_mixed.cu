// jne_accum_mixed.cu -- the mixed-precision accumulation kernels budgeted for 4
// blocks per SM (128 registers a thread), the ragged batch kernel and the
// launch dispatch.  The device code is in jne_accum_mixed.cuh; the
// 6-blocks-per-SM variants are compiled in jne_accum_mixed_b6.cu and the
// explicit-increment ones in jne_accum_mixed_ext.cu (translation units built
// in parallel).
#include "jne_accum_mixed.cuh"

namespace {

// A ragged batch of requests (any dims, step counts and sizes) in one
// persistent launch: each warp takes the next unit of the flattened batch from
// a global counter, so long and short requests share the GPU without tails.
// reqs[r].first counts units.
__device__ __forceinline__ int request_of(const jne_ragged_req* __restrict__ reqs, int n_req, long long item) {
  int lo = 0, hi = n_req - 1;  // request r with reqs[r].first <= item < reqs[r + 1].first
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (reqs[mid].first <= item) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One unit of a request, its dim's slot table written first where the warp held another dim's.
template <int DIM>
__device__ __forceinline__ void ragged_unit(const jne_accum_args& a, int unit, WarpSmem& sm, uint2* slot, int& slot_dim,
                                            const jne_round_keys& rk, int lane) {
  if (slot_dim != DIM) {
    fill_product_slots<DIM, true>(slot, lane, JNE_WARP);
    __syncwarp();
    slot_dim = DIM;
  }
  accum_unit<DIM, false, false, true>(a, unit, sm, slot, rk, lane);
}

// batch_done (ceil(total / 32) zeroed counts): every item is also finalized
// in the launch, batches of 32 consecutive items spanning requests as needed.
__global__ void __launch_bounds__(kMixWarps * JNE_WARP, 4)
    k_accum_mixed_ragged(const jne_ragged_req* __restrict__ reqs, int n_req, long long total,
                         unsigned long long* __restrict__ counter, unsigned int* __restrict__ batch_done) {
  __shared__ WarpSmem sm_all[kMixWarps];
  __shared__ uint2 slot_all[kMixWarps][kProductSlots];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int slot_dim = 0;  // the dim this warp's slot table was built for
  // first item by warp, then the next free one from the counter: the warps of a block run the same dim's code
  // (the launch's items are ordered by dim), which fits the instruction cache where several dims' does not
  const unsigned long long nwarps = (unsigned long long)gridDim.x * kMixWarps;
  for (unsigned long long item = (unsigned long long)blockIdx.x * kMixWarps + wib;
       item < (unsigned long long)total;) {
    const int lo = request_of(reqs, n_req, (long long)item);
    const jne_accum_args& a = reqs[lo].acc;
    const int unit = (int)(item - (unsigned long long)reqs[lo].first);
    const jne_round_keys rk = jne_make_round_keys(a.key0, a.key1);
    switch (a.dim) {
      case 1: ragged_unit<1>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 2: ragged_unit<2>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 3: ragged_unit<3>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 4: ragged_unit<4>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 5: ragged_unit<5>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 6: ragged_unit<6>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 7: ragged_unit<7>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 8: ragged_unit<8>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 9: ragged_unit<9>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 10: ragged_unit<10>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      case 11: ragged_unit<11>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
      default: ragged_unit<12>(a, unit, sm_all[wib], slot_all[wib], slot_dim, rk, lane); break;
    }
    if (batch_done) {
      const long long first = batch_complete(batch_done, (long long)item, total, lane);
      if (first >= 0) {
        // one run per lane; batches of packed pairs in two rounds of 16 items, batches that mix packed and
        // unpacked dims one item per lane
        const bool mine = first + lane < total;
        const int r0 = mine ? request_of(reqs, n_req, first + lane) : 0;
        const bool packed = !mine || reqs[r0].acc.dim <= JNE_PACK_MAX_DIM;
        if (__all_sync(0xffffffffu, packed)) {
          for (int s = lane; s < 64; s += 32) {
            const long long it = first + (s >> 1);
            if (it < total) {
              const jne_ragged_req& q = reqs[request_of(reqs, n_req, it)];
              const long long run = 2 * (it - q.first) + (s & 1);
              if (run < q.fin.n_runs) jne_fin::finalize_run<false>(q.fin, (int)run);
            }
          }
        } else if (mine) {
          const jne_ragged_req& q = reqs[r0];
          const int nu = packed ? 2 : 1;
          for (int u = 0; u < nu; u++) {
            const long long run = nu * (first + lane - q.first) + u;
            if (run < q.fin.n_runs) jne_fin::finalize_run<false>(q.fin, (int)run);
          }
        }
      }
      __syncwarp();
    }
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(counter, 1ull);
    item = nwarps + __shfl_sync(0xffffffffu, next, 0);
  }
}

}  // namespace

cudaError_t jne_launch_accum_mixed_ragged(const jne_ragged_req* reqs, int n_req, long long total,
                                         unsigned long long* counter, unsigned int* batch_done, int sms,
                                         cudaStream_t st) {
  if (total <= 0) return cudaSuccess;
  const int threads = kMixWarps * JNE_WARP;
  k_accum_mixed_ragged<<<resident_grid(k_accum_mixed_ragged, threads, 0, sms, total, kMixWarps), threads, 0, st>>>(
      reqs, n_req, total, counter, batch_done);
  return cudaGetLastError();
}

cudaError_t jne_launch_accum_mixed(const jne_accum_args& a, const jne_finalize_args* fin, int sms, cudaStream_t st) {
  if (a.blocks_per_sm != 0 && a.blocks_per_sm != 4 && a.blocks_per_sm != 6) return cudaErrorInvalidValue;
  if (a.ext) return jne_launch_accum_mixed_ext(a, fin, sms, st);
  if (a.blocks_per_sm == 6) return jne_launch_accum_mixed_b6(a, fin, sms, st);
  return launch_mixed<4, false>(a, fin, sms, st);
}
