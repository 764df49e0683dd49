// jne_quantile.cu -- device quantile analyzer.
//
// Replaces calculate_percentiles (simulation_analyzers.rs:42-65): the Sum or
// Max aggregate of every run's eigenvalues (:26-39), then the percentiles with
// the interpolation rule of get_percentile_value (:4-18).  The reference sorts
// all aggregates; only the two order statistics around each rank p (n - 1) are
// needed, so they are found by a most-significant-digit select on
// order-preserving 64-bit keys less their minimum: a first histogram of up to
// 2048 bins over the keys' actual range, then 128 bins a pass over each wanted rank's
// bin (where many keys share it, over the range that the last pass found them in), until
// that range is one key (tied values) or a bin holds at most 64 keys, which the next pass
// lists.  The selected keys are exact aggregate values, and the interpolation runs on the
// host with the reference's arithmetic, so the result is bit-identical to a full sort.
//
// What bounds it: for 10^6 runs of 12 values the 96 MB read (15 us at the copy
// bandwidth) and, for the sums, the FP64 additions (19 us); the passes read 8 MB of
// keys from L2, and all but the first take a key to its ranks (mostly none) by a table of
// the first bins.  Each pass's last block picks the bins and clears the counters, so a
// pass is one launch; three resolve distinct values, and the host starts more only
// when they did not.  10^6 x 12, seven percentiles: 444 us before (eight passes of
// three launches, each comparing every key with every rank's prefix), 121 now, of
// which 69 are what a call of 100 rows takes (four launches, a copy and the waits).
#include <cfloat>
#include <cstring>
#include "jne_context.h"

using namespace jne_detail;

namespace {

constexpr int kQThreads = 256;
constexpr int kPassThreads = 512;
constexpr int kGroup = 16;      // ranks per select group
constexpr int kFirstMax = 2048;  // bins of the first pass
constexpr int kSubBits = 7, kSub = 1 << kSubBits;
constexpr int kList = kSub / 2;  // keys that fit a rank's counters

// Order-preserving map of doubles to unsigned keys: negative values flip all
// bits, non-negative values set the sign bit.
__device__ __forceinline__ unsigned long long key_of(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

double value_of(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
  double v;
  std::memcpy(&v, &b, sizeof v);
  return v;
}

// Select state in device memory, ahead of the per-rank arrays.
struct QHead {
  unsigned int n_nan, ticket;
  unsigned long long neg_min, max;  // ~smallest and largest key (both start at 0)
  unsigned long long todo;          // ranks of the group still open (bit per rank)
};
constexpr int kHeadWords = sizeof(QHead) / 8 + 1;  // and the shift
constexpr int kRankWords = 6;                      // arrays per rank

// The scratch after the keys.
struct QLayout {
  QHead* head;
  unsigned int* shift;         // bits below the first digit
  unsigned long long* lo;      // per rank: its bin's first key; the rank's own key once closed
  unsigned long long* hi;      // per rank: its bin's last key
  unsigned long long* rank;    // per rank: rank within its bin
  unsigned long long* count;   // per rank: keys in its bin, twice (high and low half)
  unsigned long long* nmin;    // per rank: ~smallest and largest key found in its bin (both start at 0)
  unsigned long long* max;
  unsigned int* hist;          // bins of the current pass (kSub per rank after the first), or a small bin's keys
};

struct QRanks {
  unsigned long long r[kGroup];
};

// First-pass bins for a group of nr ranks: what keeps the scratch within 256
// counters a rank.
int first_bins(int nr) {
  int b = kSub;
  while (2 * b <= 256 * nr - 64 && 2 * b <= kFirstMax) b *= 2;
  return b;
}

// Sum (in index order, as the reference's iterator sum) or max (folded from
// f64::MIN, NaN ignored) of each run's k eigenvalues, as keys, with their
// smallest and largest; counts NaN aggregates.
// Values of a row are loaded eight at a time ahead of their (sequential) use.
template <bool PAIRS>
__global__ void __launch_bounds__(kQThreads) k_aggregate(const double* __restrict__ eigs, long long n, int k, int stat,
                                                         unsigned long long* __restrict__ keys, QHead* head) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long lo = ~0ull, hi = 0ull;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
    const double* e = eigs + r * k;
    unsigned long long key = key_of(-DBL_MAX);
    double a = 0.0;
    for (int j0 = 0; j0 < k; j0 += 8) {
      double v[8];
      if (PAIRS) {
#pragma unroll
        for (int j = 0; j < 8; j += 2)
          if (j0 + j < k) {
            const double2 p = *reinterpret_cast<const double2*>(e + j0 + j);
            v[j] = p.x;
            v[j + 1] = p.y;
          }
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j0 + j < k) v[j] = e[j0 + j];
      }
      if (stat == 0) {
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j0 + j < k) a = __dadd_rn(a, v[j]);
      } else {  // max on the keys, without FP64 instructions (beyond the infinities' keys lie NaNs)
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j0 + j < k) {
            const unsigned long long c = key_of(v[j]);
            if (c > key && c <= 0xFFF0000000000000ull) key = c;
          }
      }
    }
    if (stat == 0) {
      if (a != a) atomicAdd(&head->n_nan, 1u);
      key = key_of(a);
    }
    keys[r] = key;
    lo = min(lo, key);
    hi = max(hi, key);
  }
  for (int o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  __shared__ unsigned long long wl[kQThreads / 32], wh[kQThreads / 32];
  if ((threadIdx.x & 31) == 0) {
    wl[threadIdx.x >> 5] = lo;
    wh[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kQThreads / 32; w++) {
      lo = min(lo, wl[w]);
      hi = max(hi, wh[w]);
    }
    atomicMax(&head->neg_min, ~lo);
    atomicMax(&head->max, hi);
  }
}

// True for the threads of the last block to arrive, which sees every other
// block's writes.
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Executed by a warp: the bin of `hist` (in shared memory, a multiple of 32 bins)
// that holds rank r; r becomes the rank within it, cnt its count.
__device__ __forceinline__ int pick(const unsigned int* hist, int bins, unsigned long long& r, unsigned long long& cnt) {
  const int lane = threadIdx.x & 31, per = bins / 32;
  unsigned long long mine = 0;
  for (int b = 0; b < per; b++) mine += hist[lane * per + b];
  unsigned long long incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  // the first lane whose inclusive count exceeds r
  const int src = __ffs(__ballot_sync(0xffffffffu, incl > r)) - 1;
  int bin = 0;
  unsigned long long rr = r, c = 0;
  if (lane == src) {
    rr -= incl - mine;
    for (bin = lane * per;; bin++) {
      c = hist[bin];
      if (rr < c) break;
      rr -= c;
    }
  }
  r = __shfl_sync(0xffffffffu, rr, src);
  cnt = __shfl_sync(0xffffffffu, c, src);
  return __shfl_sync(0xffffffffu, bin, src);
}

// f(key, valid) for every key, by whole warps, four keys a lane loaded ahead.
template <typename F>
__device__ __forceinline__ void for_keys(const unsigned long long* __restrict__ keys, long long n, F&& f) {
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * kPassThreads * 4;
  for (long long base = ((long long)blockIdx.x * kPassThreads + threadIdx.x - lane) * 4; base < n; base += stride) {
    unsigned long long v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = base + 32 * u + lane < n ? keys[base + 32 * u + lane] : 0ull;
#pragma unroll
    for (int u = 0; u < 4; u++) f(v[u], base + 32 * u + lane < n);
  }
}

// First pass of a group: a histogram over the keys' range, then every rank's bin.
__global__ void __launch_bounds__(kPassThreads) k_select_first(const unsigned long long* __restrict__ keys, long long n,
                                                              int bins, int nr, const __grid_constant__ QRanks ranks,
                                                              const __grid_constant__ QLayout q) {
  __shared__ unsigned int sh[kFirstMax];
  const unsigned long long kmin = ~q.head->neg_min, range = q.head->max - kmin;
  const int bits = 64 - __clzll((long long)range);
  const int s1 = max(0, bits - (31 - __clz(bins)));
  for (int i = threadIdx.x; i < bins; i += kPassThreads) sh[i] = 0;
  __syncthreads();
  for_keys(keys, n, [&](unsigned long long key, bool valid) {
    if (valid) atomicAdd(&sh[(key - kmin) >> s1], 1u);
  });
  __syncthreads();
  for (int i = threadIdx.x; i < bins; i += kPassThreads)
    if (sh[i]) atomicAdd(&q.hist[i], sh[i]);
  if (!last_block(&q.head->ticket)) return;
  for (int i = threadIdx.x; i < bins; i += kPassThreads) sh[i] = __ldcg(&q.hist[i]);
  __syncthreads();
  const int w = threadIdx.x >> 5;
  if (w < nr) {
    unsigned long long r = ranks.r[w], c;
    const int b = pick(sh, bins, r, c);
    if ((threadIdx.x & 31) == 0) {
      const unsigned long long at = (unsigned long long)b << s1;
      q.lo[w] = kmin + at;
      q.hi[w] = kmin + min(range, at + ((1ull << s1) - 1ull));
      q.rank[w] = r;
      q.count[w] = c << 32 | c;
      q.nmin[w] = q.max[w] = 0ull;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < max(bins, nr * kSub); i += kPassThreads) q.hist[i] = 0;
  if (threadIdx.x == 0) {
    q.head->ticket = 0;
    q.head->todo = s1 == 0 ? 0ull : (1ull << nr) - 1ull;  // without lower bits a bin is one key
    *q.shift = (unsigned int)s1;
  }
}

// A later pass: a histogram over each open rank's bin; a bin of at most kList keys is
// listed instead (in its counters' place), and the rank's key taken from the list.  Ranks
// of one bin (neighbours, as a percentile's two mostly are) share the first one's.  In a
// bin of sixteen times its share of the keys, ties or a cluster are likely: such bins are
// counted per block in shared memory (tied keys would meet at one global counter) and
// the range that their keys lie in is found too (10^6 values of three kinds, seven
// percentiles: 690 us before, 92 now).
__global__ void __launch_bounds__(kPassThreads) k_select_next(const unsigned long long* __restrict__ keys, long long n,
                                                             int bins, int nr, const __grid_constant__ QLayout q) {
  __shared__ __align__(4) unsigned short ranks_of[kFirstMax];  // of each first bin, a bit each
  __shared__ unsigned long long lo[kGroup], span[kGroup], found_min[kGroup], found_max[kGroup], left;
  __shared__ int shift[kGroup], first_of[kGroup];
  __shared__ bool small[kGroup], dense[kGroup];
  __shared__ __align__(8) unsigned int sh[kGroup * kSub];
  const unsigned long long todo = q.head->todo;
  if (todo == 0) return;  // the same for every block: an earlier launch wrote it
  const unsigned long long kmin = ~q.head->neg_min;
  const int s1 = (int)*q.shift;
  for (int i = threadIdx.x; i < bins / 2; i += kPassThreads) reinterpret_cast<unsigned int*>(ranks_of)[i] = 0;
  if (threadIdx.x < nr) {
    const int g = threadIdx.x;
    lo[g] = q.lo[g];
    span[g] = q.hi[g] - lo[g];
    shift[g] = max(0, 64 - __clzll((long long)span[g]) - kSubBits);
    small[g] = (q.count[g] >> 32) <= kList;
    dense[g] = !small[g] && (q.count[g] >> 32) > 16ull * (unsigned long long)n / (unsigned int)bins;
    found_min[g] = ~0ull;
    found_max[g] = 0ull;
    int f = 0;  // the first open rank of the same bin (ranks' bins do not overlap otherwise)
    while (f < g && !((todo >> f & 1ull) && q.lo[f] == lo[g] && q.hi[f] == q.hi[g])) f++;
    first_of[g] = f;
  }
  for (int i = threadIdx.x; i < nr * kSub; i += kPassThreads) sh[i] = 0;
  if (threadIdx.x == 0) left = todo;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int g = 0; g < nr; g++)
      if ((todo >> g & 1ull) && first_of[g] == g) ranks_of[(lo[g] - kmin) >> s1] |= (unsigned short)(1u << g);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for_keys(keys, n, [&](unsigned long long key, bool valid) {
    const unsigned int mine = valid ? ranks_of[(key - kmin) >> s1] : 0u;
    if (!__any_sync(0xffffffffu, mine != 0)) return;
    for (unsigned int some = __reduce_or_sync(0xffffffffu, mine); some; some &= some - 1u) {
      const int g = __ffs(some) - 1;
      const unsigned long long at = key - lo[g];
      const bool m = (mine >> g & 1u) && at <= span[g];
      if (!__any_sync(0xffffffffu, m)) continue;
      if (small[g]) {
        if (m) {
          const unsigned int place = atomicAdd(reinterpret_cast<unsigned int*>(&q.count[g]), ~0u) - 1u;
          reinterpret_cast<unsigned long long*>(q.hist + g * kSub)[place] = key;
        }
      } else {
        const unsigned int bin = (unsigned int)(at >> shift[g]);
        const unsigned int peers = __match_any_sync(0xffffffffu, m ? bin : 0x1000u + lane);
        if (m && lane == __ffs(peers) - 1)
          atomicAdd(dense[g] ? &sh[g * kSub + bin] : &q.hist[g * kSub + bin], (unsigned int)__popc(peers));
        if (m && dense[g]) {  // (a stale look only makes the atomic superfluous)
          if (key < *(volatile unsigned long long*)&found_min[g]) atomicMin(&found_min[g], key);
          if (key > *(volatile unsigned long long*)&found_max[g]) atomicMax(&found_max[g], key);
        }
      }
    }
  });
  __syncthreads();
  for (int i = threadIdx.x; i < nr * kSub; i += kPassThreads)
    if (dense[i / kSub] && sh[i]) atomicAdd(&q.hist[i], sh[i]);
  if (threadIdx.x < nr && found_min[threadIdx.x] <= found_max[threadIdx.x]) {
    atomicMax(&q.nmin[threadIdx.x], ~found_min[threadIdx.x]);
    atomicMax(&q.max[threadIdx.x], found_max[threadIdx.x]);
  }
  if (!last_block(&q.head->ticket)) return;
  for (int i = threadIdx.x; i < nr * kSub; i += kPassThreads) {
    sh[i] = __ldcg(&q.hist[i]);
    q.hist[i] = 0;
  }
  // what the bin's first rank counted, ahead of that rank's warp writing its next bin
  const int w = threadIdx.x >> 5, f = w < nr ? first_of[w] : 0;
  const unsigned long long least = ~__ldcg(&q.nmin[f]), most = __ldcg(&q.max[f]);
  const int c_list = (int)(__ldcg(&q.count[f]) >> 32);
  __syncthreads();
  if (w < nr && (todo >> w & 1ull)) {
    unsigned long long r = q.rank[w];
    if (small[w]) {  // the key with r others before it (equal keys in list order)
      const unsigned long long* list = reinterpret_cast<const unsigned long long*>(sh + f * kSub);
      for (int i = lane; i < c_list; i += 32) {
        const unsigned long long x = list[i];
        unsigned long long before = 0;
        for (int j = 0; j < c_list; j++) {
          const unsigned long long y = list[j];
          before += y < x || (y == x && j < i);
        }
        if (before == r) q.lo[w] = x;
      }
      if (lane == 0) atomicAnd(&left, ~(1ull << w));
    } else {
      unsigned long long c;
      const int b = pick(sh + f * kSub, kSub, r, c);
      if (lane == 0) {
        // the picked bin, as far as keys were found in it
        const unsigned long long at = (unsigned long long)b << shift[w];
        unsigned long long first = lo[w] + at, last = lo[w] + min(span[w], at + ((1ull << shift[w]) - 1ull));
        if (dense[w]) {
          first = max(first, least);
          last = min(last, most);
        }
        q.lo[w] = first;
        q.hi[w] = last;
        q.rank[w] = r;
        q.count[w] = c << 32 | c;
        q.nmin[w] = q.max[w] = 0ull;
        if (first == last) atomicAnd(&left, ~(1ull << w));
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    q.head->ticket = 0;
    q.head->todo = left;
  }
}

}  // namespace

extern "C" int jne_percentiles_device(jne_context* c, const double* eigs_device, int64_t n, int k, int stat,
                                      const double* ps, int np, double* out, void* stream) {
  if (!c) return JNE_ERR_ARG;
  if ((n > 0 && !eigs_device) || (np > 0 && (!ps || !out)) || k < 1 || n < 0 || np < 0 || (stat != 0 && stat != 1))
    return fail(c, JNE_ERR_ARG, "bad percentile arguments");
  for (int i = 0; i < np; i++)
    if (!(ps[i] >= 0.0 && ps[i] <= 1.0)) return fail(c, JNE_ERR_ARG, "percentiles must lie in [0, 1]");
  if (np == 0) return JNE_OK;
  if (n == 0) {
    for (int i = 0; i < np; i++) out[i] = NAN;
    return JNE_OK;
  }
  if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, JNE_ERR_CUDA, "cudaSetDevice failed");
  int rc = drain(c);
  if (rc) return rc;
  if ((rc = join_in(c, (cudaStream_t)stream))) return rc;
  // the distinct ranks floor / ceil of p (n - 1)
  std::vector<unsigned long long> ranks;
  for (int i = 0; i < np; i++) {
    const double rank = ps[i] * (double)(n - 1);
    ranks.push_back((unsigned long long)std::floor(rank));
    ranks.push_back((unsigned long long)std::ceil(rank));
  }
  std::sort(ranks.begin(), ranks.end());
  ranks.erase(std::unique(ranks.begin(), ranks.end()), ranks.end());
  const int nr = (int)ranks.size();
  // scratch: keys | head, shift | the arrays per rank of a group | histogram
  const int ngmax = std::min(nr, kGroup), bins = first_bins(ngmax);
  const size_t hist_words = (size_t)std::max(bins, ngmax * kSub) / 2;
  const size_t words = (size_t)n + kHeadWords + kRankWords * (size_t)ngmax + hist_words;
  if ((rc = ensure(c, &c->d_qscratch, &c->qscratch_cap, words, "percentile scratch"))) return rc;
  unsigned long long* keys = c->d_qscratch;
  QLayout q;
  q.head = reinterpret_cast<QHead*>(keys + n);
  q.shift = reinterpret_cast<unsigned int*>(keys + n + kHeadWords - 1);
  q.lo = keys + n + kHeadWords;  // read back with the head
  q.hi = q.lo + ngmax;
  q.rank = q.hi + ngmax;
  q.count = q.rank + ngmax;
  q.nmin = q.count + ngmax;
  q.max = q.nmin + ngmax;
  q.hist = reinterpret_cast<unsigned int*>(q.max + ngmax);
  cudaStream_t st = c->stream;
  cudaError_t e = cudaMemsetAsync(keys + n, 0, sizeof(unsigned long long) * (words - (size_t)n), st);
  if (e != cudaSuccess) return cuda_fail(c, e, "percentile setup");
  const long long want = (n + kQThreads - 1) / kQThreads;
  const int grid = (int)std::min<long long>(want, (long long)c->sms * 8);
  // even rows of a 16-byte aligned table in 16-byte loads
  if (k % 2 == 0 && reinterpret_cast<uintptr_t>(eigs_device) % 16 == 0)
    k_aggregate<true><<<grid, kQThreads, 0, st>>>(eigs_device, n, k, stat, keys, q.head);
  else
    k_aggregate<false><<<grid, kQThreads, 0, st>>>(eigs_device, n, k, stat, keys, q.head);
  const long long want_pass = (n + 4 * kPassThreads - 1) / (4 * kPassThreads);  // four keys a thread and round
  const int grid_pass = (int)std::min<long long>(want_pass, (long long)c->sms * 2);
  std::vector<unsigned long long> sel(nr), back(kHeadWords + (size_t)ngmax);
  unsigned int nans = 0;
  for (int g0 = 0; g0 < nr; g0 += kGroup) {
    const int ng = std::min(kGroup, nr - g0);
    QRanks gr{};
    for (int g = 0; g < ng; g++) gr.r[g] = ranks[(size_t)(g0 + g)];
    k_select_first<<<grid_pass, kPassThreads, 0, st>>>(keys, n, bins, ng, gr, q);
    unsigned long long todo = 1;
    // at most 57 bits below the first digit, 7 a pass, and one more for a rank alone in its bin
    for (int pass = 0; pass < 10 && todo; pass += 2) {
      k_select_next<<<grid_pass, kPassThreads, 0, st>>>(keys, n, bins, ng, q);
      k_select_next<<<grid_pass, kPassThreads, 0, st>>>(keys, n, bins, ng, q);
      e = cudaGetLastError();
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(back.data(), q.head, sizeof(unsigned long long) * (kHeadWords + (size_t)ng),
                            cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) return cuda_fail(c, e, "percentile select");
      QHead head;
      std::memcpy(&head, back.data(), sizeof head);
      todo = head.todo;
      nans = head.n_nan;
    }
    for (int g = 0; g < ng; g++) sel[(size_t)(g0 + g)] = back[kHeadWords + (size_t)g];
  }
  if (nans) return fail(c, JNE_ERR_NUMERIC, std::to_string(nans) + " runs have a NaN aggregate (unordered)");
  auto at = [&](unsigned long long r) {
    const size_t i = (size_t)(std::lower_bound(ranks.begin(), ranks.end(), r) - ranks.begin());
    return value_of(sel[i]);
  };
  for (int i = 0; i < np; i++) {  // get_percentile_value, simulation_analyzers.rs:4-18
    const double rank = ps[i] * (double)(n - 1);
    const unsigned long long lo = (unsigned long long)std::floor(rank), hi = (unsigned long long)std::ceil(rank);
    if (lo == hi) {
      out[i] = at(lo);
    } else {
      const double wgt = rank - (double)lo;
      out[i] = at(lo) * (1.0 - wgt) + at(hi) * wgt;
    }
  }
  return JNE_OK;
}
