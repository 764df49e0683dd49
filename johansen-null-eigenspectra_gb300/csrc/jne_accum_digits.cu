// jne_accum_digits.cu -- launches of the FP64 accumulation in exact digits
// (jne_accum_digits.cuh) for the engine's own increments, dims 1..6; the larger
// dims are compiled in jne_accum_digits_hi.cu (translation units built in
// parallel), and of paths too short for digits.  Explicit increments, whose range and precision are the caller's,
// keep the kernel of jne_accum_f64.cu.
#include "jne_accum_digits.cuh"

namespace {

// Paths of at most JNE_SHORT_STEPS (one tile): FP64 multiply-adds, one warp per run.  On so few steps S11 is close
// to singular and the pencil magnifies what the digits leave out (dim 12, T 17, model 0, rms against quad precision:
// digits 2.1e-14, multiply-adds 0.9e-14; dim 8, T 10: 2.3e-11, 1.1e-12; equal near T 30).  Lane t draws step t, feature
// f's lanes walk it, and every lane sums its <= 9 products v_t[a] v_t[b], v_t = [W; z; 1; y; y^2], of the
// moments the model needs.  Bound by the FP64 pipe: 20,000 runs at dim 12, T 32, model 1 1.49 ms (digits 1.20, separate
// accumulation and finalize kernels 1.57); 100,000 at dim 2 0.31 (0.34, 0.44).
constexpr int kShortEntries = 9;             // (78 + 144 + 5 * 12) / 32 at dim 12
constexpr int kVS = 2 * JNE_MAX_DIM + 5;     // odd row stride: conflict-free column writes

// N entries per lane: counted out, because an FP64 instruction holds its pipe even when predicated off.
template <int N>
__device__ __forceinline__ void sum_products(const double (*v)[kVS], int T, const int (&op)[kShortEntries],
                                             double (&acc)[kShortEntries]) {
  for (int t = 0; t < T; t++)
#pragma unroll
    for (int m = 0; m < N; m++) acc[m] = fma(v[t][op[m] & 0xff], v[t][op[m] >> 8], acc[m]);
}

__global__ void __launch_bounds__(kMixWarps * JNE_WARP)
    k_accum_short(const __grid_constant__ jne_accum_args a, const __grid_constant__ jne_round_keys rk,
                  const __grid_constant__ jne_finalize_args fin) {
  __shared__ double v_all[kMixWarps][JNE_SHORT_STEPS][kVS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int d = a.dim, T = a.steps, kinds = moment_kinds(a.model), one = 2 * d;
  const int nb = a.model == 2 || a.model == 4 ? d - 1 : d;  // walk rows that enter F
  const int nww = nb * (nb + 1) / 2, nprod = nww + d * nb;
  const int ne = nprod + (kinds > 0 ? nb : 0) + (kinds > 1 ? nb + d : 0) + (kinds > 3 ? nb + d : 0);
  double (*v)[kVS] = v_all[wib];
  for (int e = lane; e < JNE_SHORT_STEPS * kVS; e += JNE_WARP) (&v[0][0])[e] = 0.0;  // rows past T stay zero
  __syncwarp();
  int seg = 1;  // lanes that share a feature's walk (a power of two)
  while (2 * seg * d <= JNE_WARP) seg *= 2;
  const int wf = lane / seg, wq = lane - wf * seg, len = JNE_SHORT_STEPS / seg;
  const double invT = 1.0 / (double)T;
  const int nwarps = gridDim.x * kMixWarps;
  const bool fused = fin.out != nullptr && a.batch_done != nullptr;
  int op[kShortEntries], slot[kShortEntries];
#pragma unroll
  for (int m = 0; m < kShortEntries; m++) {
    const int e = lane + JNE_WARP * m;
    int x = 0, y = 0;
    slot[m] = -1;
    if (e < nww) {
      int p = 0, r = e;
      while (r >= nb - p) { r -= nb - p; p++; }
      x = p; y = p + r; slot[m] = jne_slot_MWW(x, y, d);
    } else if (e < nprod) {
      const int r = e - nww, za = r / nb, wb = r - za * nb;
      x = d + za; y = wb; slot[m] = jne_slot_NzW(za, wb, d);
    } else if (e < ne) {  // W | y W, y z | y^2 W, y^2 z
      int kind = 0, f = e - nprod;
      for (int n = nb; f >= n; n = kind == 2 || kind == 4 ? d : nb) { f -= n; kind++; }
      const int p = (kind + 1) >> 1;
      const bool inc = kind == 2 || kind == 4;
      x = inc ? d + f : f; y = one + p;
      slot[m] = inc ? (p == 1 ? jne_slot_Nzy(f, d) : jne_slot_Nzyy(f, d))
                    : p == 0 ? jne_slot_MW1(f, d) : p == 1 ? jne_slot_MWy(f, d) : jne_slot_MWyy(f, d);
    }
    op[m] = x | y << 8;
  }
  for (long long run = blockIdx.x * kMixWarps + wib; run < a.n_runs;) {
    if (lane < T) {
      double* row = v[lane];
      for (int j = 0; 4 * j < d; j++) {
        float z[4];
        jne_normal_quad((uint32_t)(lane + 1), (uint32_t)j, a.seed_first + (uint32_t)run, rk, z);
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (4 * j + e < d) row[d + 4 * j + e] = (double)z[e];
      }
      const double y = (double)(lane + 1) * invT;
      row[one] = 1.0;
      row[one + 1] = y;
      row[one + 2] = y * y;
    }
    __syncwarp();
    double sum = 0.0;  // the walk: each lane's segment, an exclusive scan of the segments, the segment again
    if (wf < d)
      for (int t = 0; t < len; t++) sum += v[wq * len + t][d + wf];
    for (int o = 1; o < seg; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, sum, o, seg);
      if (wq >= o) sum += up;
    }
    const double before = __shfl_up_sync(0xffffffffu, sum, 1, seg);
    double W = wq > 0 ? before : 0.0;
    if (wf < d)
      for (int t = 0; t < len; t++) {
        v[wq * len + t][wf] = W;
        W += v[wq * len + t][d + wf];
      }
    __syncwarp();
    double acc[kShortEntries];
#pragma unroll
    for (int m = 0; m < kShortEntries; m++) acc[m] = 0.0;
    switch ((ne + JNE_WARP - 1) / JNE_WARP) {
      case 1: sum_products<1>(v, T, op, acc); break;
      case 2: sum_products<2>(v, T, op, acc); break;
      case 3: sum_products<3>(v, T, op, acc); break;
      case 4: sum_products<4>(v, T, op, acc); break;
      case 5: sum_products<5>(v, T, op, acc); break;
      case 6: sum_products<6>(v, T, op, acc); break;
      case 7: sum_products<7>(v, T, op, acc); break;
      case 8: sum_products<8>(v, T, op, acc); break;
      default: sum_products<9>(v, T, op, acc); break;
    }
#pragma unroll
    for (int m = 0; m < kShortEntries; m++)
      if (slot[m] >= 0) a.mom[(size_t)slot[m] * a.mom_ld + run] = acc[m];
    if (wf < d && wq == seg - 1) a.mom[(size_t)jne_slot_Nz1(wf, d) * a.mom_ld + run] = W;
    if (fused) {
      const long long first = batch_complete(a.batch_done, run, a.n_runs, lane);
      if (first >= 0) finalize_batch(fin, first, false, lane);
    }
    __syncwarp();
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(a.next_run, 1ull);
    run = nwarps + (long long)__shfl_sync(0xffffffffu, item, 0);
  }
}

}  // namespace

cudaError_t jne_launch_accum_digits(const jne_accum_args& a, const jne_finalize_args* fin, int sms, cudaStream_t st) {
  if (a.n_runs <= 0) return cudaSuccess;
  if (a.ext || !a.next_run) return cudaErrorInvalidValue;
  jne_finalize_args f{};  // out == nullptr: accumulation only
  if (fin) f = *fin;
  if (a.steps <= JNE_SHORT_STEPS) {
    const int threads = kMixWarps * JNE_WARP;
    k_accum_short<<<resident_grid(k_accum_short, threads, 0, sms, a.n_runs, kMixWarps), threads, 0, st>>>(
        a, jne_make_round_keys(a.key0, a.key1), f);
    return cudaGetLastError();
  }
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
