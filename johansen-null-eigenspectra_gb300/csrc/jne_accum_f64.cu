// jne_accum_f64.cu -- FP64 accumulation of explicit increments: one warp per run.
//
// Replaces, per run, the work of johansen_statistics.rs:102-197 (F
// construction) and the two sum_of_outer_products calls of
// johansen_statistics.rs:32-33: instead of materialising B and F, each run
// accumulates in FP64 multiply-adds the raw moments its model needs (listed in a
// per-(model, dim) entry table), from which the finalize kernel rebuilds S11 and
// S10.  The engine's own increments take jne_accum_digits.cuh, whose fixed-point
// grid an arbitrary FP64 increment does not fit.
//
// Per 32-step tile: lane t reads the increments of column t0+t, the lanes run the
// FP64 walk along time (two passes of 32 / seg additions in seg lanes per feature:
// 11 additions a tile at dim 4, where one lane per feature took 32), and every lane
// adds its <= MAXE table entries sum_t v_t[a] * v_t[b] over the tile, where
// v_t = [W_0..W_{d-1}, z_0..z_{d-1}, 1, y, y^2, 0].  Bound by the FP64 pipe (64
// cycles a warp instruction and scheduler): 2,000 runs at dim 4, T 1000, the 64 MB
// upload included, 839 us with one lane per feature walking, 671 now; 20,000 runs at
// dim 2 4.36 -> 3.51 ms.
#include "jne_common.cuh"
#include "jne_kernels.h"

namespace {

constexpr int kF64Warps = 4;  // warps per block

template <int MAXE>
__global__ void __launch_bounds__(kF64Warps * JNE_WARP)
    k_accum_f64(const jne_accum_args a, const int4* __restrict__ ent, const int nent) {
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int d = a.dim, T = a.steps;
  const int VS = 2 * d + 5;  // odd row stride: conflict-free column writes
  const int ZERO = 2 * d + 3;
  int seg = 1;  // lanes that share a feature's walk (a power of two)
  while (2 * seg * d <= JNE_WARP) seg *= 2;
  double* v = smem + (size_t)wib * JNE_WARP * VS;
  for (int e = lane; e < JNE_WARP * VS; e += JNE_WARP) v[e] = 0.0;

  int opA[MAXE], opB[MAXE], slot[MAXE];
#pragma unroll
  for (int m = 0; m < MAXE; m++) {
    const int e = lane + JNE_WARP * m;
    if (e < nent) {
      const int4 t = ent[e];
      opA[m] = t.x; opB[m] = t.y; slot[m] = t.z;
    } else {
      opA[m] = ZERO; opB[m] = ZERO; slot[m] = -1;
    }
  }
  const double invT = 1.0 / (double)T;
  const int nwarps = gridDim.x * kF64Warps;
  __syncwarp();

  for (int run = blockIdx.x * kF64Warps + wib; run < a.n_runs; run += nwarps) {
    double acc[MAXE];
#pragma unroll
    for (int m = 0; m < MAXE; m++) acc[m] = 0.0;
    double carry = 0.0;  // W_f at the tile start, in the lanes of feature f

    for (int t0 = 0; t0 < T; t0 += JNE_WARP) {
      const int i = t0 + lane;
      const bool valid = i < T;
      double* vr = v + lane * VS;
      const double* src = a.ext + ((size_t)run * T + (valid ? i : 0)) * d;
      for (int f = 0; f < d; f++) vr[d + f] = valid ? src[f] : 0.0;
      const double y = (double)(i + 1) * invT;
      vr[2 * d] = valid ? 1.0 : 0.0;
      vr[2 * d + 1] = valid ? y : 0.0;
      vr[2 * d + 2] = valid ? y * y : 0.0;
      __syncwarp();
      {  // exclusive walk W_i = sum_{s <= i} z_s along the tile: `seg` lanes per feature take 32 / seg steps each
        const int nv = min(JNE_WARP, T - t0), f = lane / seg, q = lane - f * seg, len = JNE_WARP / seg;
        double* col = v + (q * len) * VS + (f < d ? f : 0);
        double sum = 0.0;
        if (f < d)
          for (int t = 0; t < len; t++) sum += col[t * VS + d];
        double incl = sum;  // inclusive scan of the segments' sums
        for (int o = 1; o < seg; o <<= 1) {
          const double up = __shfl_up_sync(0xffffffffu, incl, o, seg);
          if (q >= o) incl += up;
        }
        const double before = __shfl_up_sync(0xffffffffu, incl, 1, seg);
        double W = q > 0 ? carry + before : carry;
        if (f < d)
          for (int t = 0; t < len; t++) {
            col[t * VS] = q * len + t < nv ? W : 0.0;
            W += col[t * VS + d];
          }
        carry = __shfl_sync(0xffffffffu, W, seg - 1, seg);
      }
      __syncwarp();
      for (int tau = 0; tau < JNE_WARP; tau++) {
        const double* vt = v + tau * VS;
#pragma unroll
        for (int m = 0; m < MAXE; m++) acc[m] = fma(vt[opA[m]], vt[opB[m]], acc[m]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int m = 0; m < MAXE; m++)
      if (slot[m] >= 0) a.mom[(size_t)slot[m] * a.mom_ld + run] = acc[m];
    if (lane % seg == 0 && lane / seg < d) a.mom[(size_t)jne_slot_Nz1(lane / seg, d) * a.mom_ld + run] = carry;
  }
}

template <int MAXE>
cudaError_t launch_maxe(const jne_accum_args& a, const int4* ent, int nent, int sms, cudaStream_t st) {
  const int VS = 2 * a.dim + 5;
  const size_t shm = (size_t)kF64Warps * JNE_WARP * VS * sizeof(double);
  const int threads = kF64Warps * JNE_WARP;
  auto k = k_accum_f64<MAXE>;
  // persistent grid: the resident blocks, so every warp strides over the same number of runs
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, shm) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  const int needed = (a.n_runs + kF64Warps - 1) / kF64Warps;
  const int grid = needed < per_sm * sms ? needed : per_sm * sms;
  k<<<grid, threads, shm, st>>>(a, ent, nent);
  return cudaGetLastError();
}

}  // namespace

cudaError_t jne_launch_accum_f64(const jne_accum_args& a, const int4* ent, int nent, int sms, cudaStream_t st) {
  if (a.n_runs <= 0) return cudaSuccess;
  if (!a.ext) return cudaErrorInvalidValue;
  switch ((nent + JNE_WARP - 1) / JNE_WARP) {
    case 1: return launch_maxe<1>(a, ent, nent, sms, st);
    case 2: return launch_maxe<2>(a, ent, nent, sms, st);
    case 3: return launch_maxe<3>(a, ent, nent, sms, st);
    case 4: return launch_maxe<4>(a, ent, nent, sms, st);
    case 5: return launch_maxe<5>(a, ent, nent, sms, st);
    case 6: return launch_maxe<6>(a, ent, nent, sms, st);
    case 7: return launch_maxe<7>(a, ent, nent, sms, st);
    case 8: return launch_maxe<8>(a, ent, nent, sms, st);
    case 9: return launch_maxe<9>(a, ent, nent, sms, st);
    default: return cudaErrorInvalidValue;
  }
}

// Entry table of a (model, dim) pair: the moments its F needs (Nz1 comes from the
// walk's end point).
int jne_build_f64_entries(int model, int d, int4* out, int cap) {
  const int W = 0, Z = d, ONE = 2 * d, Y = 2 * d + 1, YY = 2 * d + 2;
  const int nb = (model == 2 || model == 4) ? d - 1 : d;  // walk rows entering F
  const bool need_w1 = model >= 1;
  const bool need_y = model >= 2;
  const bool need_yy = model == 4;
  int n = 0;
  auto put = [&](int x, int y, int s) {
    if (n < cap) out[n] = make_int4(x, y, s, 0);
    n++;
  };
  for (int p = 0; p < nb; p++)
    for (int q = p; q < nb; q++) put(W + p, W + q, jne_slot_MWW(p, q, d));
  for (int p = 0; p < nb; p++) {
    if (need_w1) put(W + p, ONE, jne_slot_MW1(p, d));
    if (need_y) put(W + p, Y, jne_slot_MWy(p, d));
    if (need_yy) put(W + p, YY, jne_slot_MWyy(p, d));
  }
  for (int a = 0; a < d; a++)
    for (int b = 0; b < nb; b++) put(Z + a, W + b, jne_slot_NzW(a, b, d));
  for (int a = 0; a < d; a++) {
    if (need_y) put(Z + a, Y, jne_slot_Nzy(a, d));
    if (need_yy) put(Z + a, YY, jne_slot_Nzyy(a, d));
  }
  return n;
}
