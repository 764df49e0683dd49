// jne_accum_digits.cuh -- the plain (FP64) accumulation of the engine's own
// increments: one warp per run (or per pair of runs), every Gram sum exact (as
// long as it stays in the accumulators' range, below), on the tensor cores.
//
// Same contract as jne_accum_f64.cu (rng_matrix.rs:57-141, F's moments of
// johansen_statistics.rs:102-197 and the sum_of_outer_products calls of
// johansen_statistics.rs:32-33): the FP64 moment record of jne_common.cuh.
//
// The increments are FP32 numbers, so a path needs no floating-point walk: z is
// put on a fixed-point grid of 2^-(40 + sh) (exactly, but for |z| < 2^-17, whose
// last bits are rounded), and the walk relative to the chunk's start is an exact
// 64-bit integer.  It is cut into five balanced digits of base 2^10,
//     b = 2^-sh (d0 + d1 2^-10 + d2 2^-20 + d3 2^-30 + d4 2^-40),
// |d1..d4| <= 512, d0 the (signed) rest; digits are exact in FP16, a product of
// two has 18 bits, and sums of them stay exact in the tensor core's FP32
// accumulators.  A Gram entry is then sum_s 2^(-10 s) G_s with
// G_s = sum_{i+j=s} sum_t d_i d'_j, s <= 5: the pairs left out (s >= 6) weigh
// less than the rounding of an FP64 accumulation.  The chunk's sums are combined
// in 64-bit integers, rounded once to FP64, and added to the record in FP64.
//
// Accumulator range.  G_s holds integers below 2^24 exactly:
//   * d0 is bounded by ending the chunk (for any reason a chunk may end: the
//     merge takes any length) once the walk has passed jne_digit_limit, 6.8
//     standard deviations of a full chunk (a packed pair of which one run does so is
//     computed run by run, digit_pair_apart);
//   * the squares on the diagonal are the only sums that grow with the chunk's
//     length rather than its root: their expectation, (1024^2 - 1) / 12 a step
//     for uniform digits, is taken out of the accumulator tile by tile and put
//     back at the chunk's end.  What remains is a random walk of standard
//     deviation 2^16.3 a step: 2^20.8 after 512 steps.
// Past the range a sum would only be rounded to FP32.
//
// Symmetry.  Of the walk x walk block (i, j) and (j, i) are each other's
// transposes, so only i < j is formed (and half of i = j), and the merge adds
// the transpose: 11 digit pairs instead of 19.  Increment columns need all of
// theirs; an increment's fifth digit (|z| < 2^-15 only) is formed when a tile
// has one.
//
// Why: FP64 instructions take 64 cycles a warp and scheduler on this GPU, an
// m16n8k16 MMA (2048 products) 8.  Dim 12, T 10^4, model 4, 10,000 runs: 50.8 ms
// with FP64 multiply-adds (one warp per run, 7-9 table entries per lane), 5.78 ms
// in digits; dim 5, T 1000, 50,001 runs: 9.62 -> 1.94 ms.  Errors against quad
// precision (normwise, rms over runs, dim 12): model 1, T 10^4 2.6e-12 -> 9.3e-15,
// T 1000 5.5e-14 -> 7.8e-15, T 33 6.2e-15 -> 4.4e-15; shorter paths keep the
// multiply-adds (jne_accum_digits.cu).
// What bounds it now: 94 MMAs per 32-step tile (752 cycles; 2 more for half a tile that
// has an increment with a fifth digit, about one in 300), beside which the digit
// extraction's integer instructions (2 cycles each) and the Philox multiplies (3.3)
// hardly run.  Registers: 72 accumulators; 3 blocks of 4 warps per SM (168
// registers) measured 5.7 ms of accumulation, 2 blocks (255) 5.8, 4 blocks (128,
// spilling) 6.3.
#pragma once
#include "jne_accum_mixed.cuh"

namespace {

constexpr int kDig = 5;              // digits of a walk value
constexpr int kGroups = 6;           // G_0 .. G_5
constexpr int kCD = 29;              // chunk-Gram staging row stride (doubles)
constexpr float kSquareMean = 2796200.0f;  // 32 (1024^2 - 1) / 12: a tile's expected sum of squares of a digit
constexpr long long kDigBias = 512ll * (1ll + (1ll << 10) + (1ll << 20) + (1ll << 30));

// Steps per chunk and the scale 2^sh of its digits by path length: short paths
// take finer digits (their moments are smaller) and shorter chunks (so that the
// finer digits keep their range).
__host__ __device__ __forceinline__ int jne_digit_chunk(int steps) { return steps > 2048 ? 512 : steps > 512 ? 256 : 128; }
__host__ __device__ __forceinline__ int jne_digit_shift(int steps) { return steps > 2048 ? 0 : steps > 512 ? 1 : 2; }
// |d0| beyond which a chunk ends
__host__ __device__ __forceinline__ int jne_digit_limit(int steps) { return steps > 2048 ? 154 : steps > 512 ? 218 : 309; }

struct alignas(16) DigSmem {
  float zs[16][kZS];          // increments of the current tile
  uint32_t basis[5][16];      // FP16 pairs at the tile's steps: 0, 1, c, c^2 = 1024 eA + eB (c = step - chunk centre)
  double cm[16][kCD];         // the chunk's local Gram
  double wc[16], tz[16];      // walk at the chunk start, chunk increment totals
  double sb[16], sw[16];      // sums of b and of W over the chunk
  double rec[kRecMax];
  unsigned short mww_pr[JNE_MAX_DIM * (JNE_MAX_DIM + 1) / 2];
};

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }

// Two 10-bit fields (bits 0..9 and 16..25 of u) as balanced FP16 digits: the
// field in the mantissa of 1024 + field, less 1536.
__device__ __forceinline__ uint32_t balanced(uint32_t u) {
  return h2_bits(__hadd2(bits_h2((u & 0x03FF03FFu) | 0x64006400u), __floats2half2_rn(-1536.f, -1536.f)));
}

// The digits of two consecutive steps' fixed-point values (bias added) as FP16 pairs.
__device__ __forceinline__ void digit_words(long long x, long long y, uint32_t (&w)[kDig]) {
  const uint32_t xl = (uint32_t)x, yl = (uint32_t)y, xh = (uint32_t)(x >> 32), yh = (uint32_t)(y >> 32);
  w[4] = balanced(__byte_perm(xl, yl, 0x5410));
  w[3] = balanced(__byte_perm(xl << 6, yl << 6, 0x7632));
  w[2] = balanced(__byte_perm(xl, yl, 0x7632) >> 4);
  w[1] = balanced(__byte_perm(__funnelshift_r(xl, xh, 30), __funnelshift_r(yl, yh, 30), 0x5410));
  w[0] = h2_bits(__floats2half2_rn((float)((int)xh >> 8), (float)((int)yh >> 8)));
}

// z on the grid 2^-Q, rounded to nearest, in units of 2^-Q / m; s = 2^(Q - 23),
// Q <= 42 (|z| <= 6.77 keeps z s below 2^22): floor(z s) from a round-down magic
// add, the fraction (exact) as a 23-bit integer.  t's bits are 0x4B400000 + floor;
// the constant times 2^23 m has no low word (m <= 64) and `top` takes it off.
struct FixedScale {
  float s;
  uint32_t m, top;
};
__device__ __forceinline__ FixedScale fixed_scale(int Q, int log2_m) {
  return {(float)(1 << (Q - 23)), 1u << log2_m, 0u - (0x4B400000u >> (9 - log2_m))};
}
__device__ __forceinline__ long long to_fixed(float z, const FixedScale& f) {
  const float t = __fmaf_rd(z, f.s, 12582912.f);
  const float r = __fmaf_rn(z, f.s, -__fsub_rn(t, 12582912.f));
  const uint32_t lo = (__float_as_uint(__fmaf_rn(r, 8388608.f, 8388608.f)) & 0x00FFFFFFu) * f.m;
  return (long long)((unsigned long long)__float_as_uint(t) * (f.m << 23) + (((unsigned long long)f.top << 32) | lo));
}

// An integer below 2^51 in magnitude as a double (one FP64 addition).
__device__ __forceinline__ double int_to_f64(long long v) {
  return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

__device__ __forceinline__ long long shfl_xor_ll(long long v, int m) {
  const uint32_t lo = __shfl_xor_sync(0xffffffffu, (uint32_t)v, m), hi = __shfl_xor_sync(0xffffffffu, (uint32_t)(v >> 32), m);
  return (long long)(((unsigned long long)hi << 32) | lo);
}

// 2^50 sum_s 2^(-10 s) G_s of one accumulator element (times k if the G_s are
// given times k), rounded once.
__device__ __forceinline__ double combine(int g0, int g1, int g2, int g3, int g4, int g5) {
  const long long hi = ((long long)g0 * 1048576ll + (long long)g1 * 1024ll) + g2;
  const long long lo = ((long long)g3 * 1048576ll + (long long)g4 * 1024ll) + g5;
  return fma(int_to_f64(hi), 0x1p30, int_to_f64(lo));
}

// One 32-step tile.
template <int DIM, bool FULL, bool PACK>
__device__ __forceinline__ void digit_tile(const float (*zs)[kZS], const uint32_t (*basis)[16], int g, int q, int nvalid,
                                           int selA, int selB, FixedScale scaleA, FixedScale scaleB, long long& carA,
                                           long long& carB, float diag0, float diag1, float (&acc)[3][kGroups][4]) {
  constexpr bool PAIR = Packing<DIM, PACK>::kPair;
  constexpr bool BLOCK1 = PAIR || DIM > 8;
  float zA[8];
  long long iA[8], iB[8];
  {
    const int ra = PAIR ? (g < 4 ? g : g + 4) : g;
    const float4 p0 = *reinterpret_cast<const float4*>(&zs[ra][8 * q]);
    const float4 p1 = *reinterpret_cast<const float4*>(&zs[ra][8 * q + 4]);
    zA[0] = p0.x; zA[1] = p0.y; zA[2] = p0.z; zA[3] = p0.w; zA[4] = p1.x; zA[5] = p1.y; zA[6] = p1.z; zA[7] = p1.w;
#pragma unroll
    for (int j = 0; j < 8; j++) iA[j] = to_fixed(zA[j], scaleA);
    if (BLOCK1) {
      const float4 r0 = *reinterpret_cast<const float4*>(&zs[8 + (g & 3)][8 * q]);
      const float4 r1 = *reinterpret_cast<const float4*>(&zs[8 + (g & 3)][8 * q + 4]);
      const float zB[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
      for (int j = 0; j < 8; j++) iB[j] = to_fixed(zB[j], scaleB);
    }
  }
  // lane totals and their exclusive scan over the 4 lanes of the group (a butterfly: integers add in any order)
  long long wA, wB = 0;
  {
    long long tA = ((iA[0] + iA[1]) + (iA[2] + iA[3])) + ((iA[4] + iA[5]) + (iA[6] + iA[7]));
    long long oA = shfl_xor_ll(tA, 1);
    wA = carA + kDigBias + ((q & 1) ? oA : 0ll);
    tA += oA;
    oA = shfl_xor_ll(tA, 2);
    wA += (q & 2) ? oA : 0ll;
    carA += tA + oA;
    if (BLOCK1) {
      long long tB = ((iB[0] + iB[1]) + (iB[2] + iB[3])) + ((iB[4] + iB[5]) + (iB[6] + iB[7]));
      long long oB = shfl_xor_ll(tB, 1);
      wB = carB + kDigBias + ((q & 1) ? oB : 0ll);
      tB += oB;
      oB = shfl_xor_ll(tB, 2);
      wB += (q & 2) ? oB : 0ll;
      carB += tB + oB;
    }
  }
  // PAIR: lanes g >= 4 hold run B's increments in zA (block 2's B operand): their A rows are basis rows only.
  // Otherwise lanes g >= 4 of block 1 hold increments 8..11: B columns, and basis rows (or none) as A rows.
  const bool walkA = !PAIR || g < 4, walkB = PAIR || g < 4;
  const uint32_t maskA = walkA ? ~0u : 0u, maskB = g < 4 ? ~0u : 0u;
#pragma unroll
  for (int s = 0; s < 2; s++) {
    uint32_t A[kDig][4], B1[kDig][2], B2[kDig][2];
    uint32_t v0 = ~0u, v1 = ~0u;  // valid steps of the two words
    if (!FULL) {
      const int j0 = 8 * q + 4 * s;
      v0 = (j0 < nvalid ? 0xFFFFu : 0u) | (j0 + 1 < nvalid ? 0xFFFF0000u : 0u);
      v1 = (j0 + 2 < nvalid ? 0xFFFFu : 0u) | (j0 + 3 < nvalid ? 0xFFFF0000u : 0u);
    }
    const uint2 bA = *reinterpret_cast<const uint2*>(&basis[selA][4 * q + 2 * s]);
    const uint2 bB = *reinterpret_cast<const uint2*>(&basis[selB][4 * q + 2 * s]);
    {  // row g
      uint32_t w0[kDig], w1[kDig];
      const long long x0 = wA, x1 = x0 + iA[4 * s], x2 = x1 + iA[4 * s + 1], x3 = x2 + iA[4 * s + 2];
      wA = x3 + iA[4 * s + 3];
      digit_words(x0, x1, w0);
      digit_words(x2, x3, w1);
#pragma unroll
      for (int i = 0; i < kDig; i++) {
        A[i][0] = PAIR ? w0[i] & maskA : w0[i];
        A[i][2] = PAIR ? w1[i] & maskA : w1[i];
        if (i == 0 && (PAIR || DIM < 8)) {
          A[0][0] |= bA.x;
          A[0][2] |= bA.y;
        }
        if (!FULL) {
          A[i][0] &= v0;
          A[i][2] &= v1;
        }
      }
    }
    {  // row g + 8 and block 1's columns
      uint32_t w0[kDig], w1[kDig];
      if (BLOCK1) {
        long long x0, x1, x2, x3;
        if (PAIR) {
          x0 = wB; x1 = x0 + iB[4 * s]; x2 = x1 + iB[4 * s + 1]; x3 = x2 + iB[4 * s + 2];
          wB = x3 + iB[4 * s + 3];
        } else {
          const long long y1 = wB + iB[4 * s], y2 = y1 + iB[4 * s + 1], y3 = y2 + iB[4 * s + 2];
          x0 = walkB ? wB : iB[4 * s] + kDigBias;
          x1 = walkB ? y1 : iB[4 * s + 1] + kDigBias;
          x2 = walkB ? y2 : iB[4 * s + 2] + kDigBias;
          x3 = walkB ? y3 : iB[4 * s + 3] + kDigBias;
          wB = y3 + iB[4 * s + 3];
        }
        digit_words(x0, x1, w0);
        digit_words(x2, x3, w1);
      }
#pragma unroll
      for (int i = 0; i < kDig; i++) {
        if (BLOCK1) {
          B1[i][0] = w0[i];
          B1[i][1] = w1[i];
          A[i][1] = w0[i] & maskB;
          A[i][3] = w1[i] & maskB;
        } else {
          A[i][1] = A[i][3] = 0u;
        }
        if (i == 0) {
          A[0][1] |= bB.x;
          A[0][3] |= bB.y;
        }
        if (!FULL) {
          A[i][1] &= v0;
          A[i][3] &= v1;
        }
      }
    }
    // increment columns of block 2: four digits of base 2^10 from 2^-8 down, and what is left
    float rest;
    {
      const float M = 12582912.f;
      float r[4], d[4];
      bool more = false;
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float t = __fmaf_rn(zA[4 * s + e], 256.f, M);
        d[e] = __fsub_rn(t, M);
        r[e] = __fmaf_rn(zA[4 * s + e], 256.f, -d[e]);
      }
      B2[0][0] = h2_bits(__floats2half2_rn(d[0], d[1]));
      B2[0][1] = h2_bits(__floats2half2_rn(d[2], d[3]));
#pragma unroll
      for (int j = 1; j < 4; j++) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
          d[e] = __fsub_rn(__fmaf_rn(r[e], 1024.f, M), M);
          r[e] = __fmaf_rn(r[e], 1024.f, -d[e]);
        }
        B2[j][0] = h2_bits(__floats2half2_rn(d[0], d[1]));
        B2[j][1] = h2_bits(__floats2half2_rn(d[2], d[3]));
      }
      rest = fmaxf(fmaxf(fabsf(r[0]), fabsf(r[1])), fmaxf(fabsf(r[2]), fabsf(r[3])));
      more = __any_sync(0xffffffffu, rest != 0.f);
      if (more) {
        B2[4][0] = h2_bits(__floats2half2_rn(r[0] * 1024.f, r[1] * 1024.f));
        B2[4][1] = h2_bits(__floats2half2_rn(r[2] * 1024.f, r[3] * 1024.f));
        mma_f16(acc[2][4], A[0][0], A[0][1], A[0][2], A[0][3], B2[4][0], B2[4][1]);
        mma_f16(acc[2][5], A[1][0], A[1][1], A[1][2], A[1][3], B2[4][0], B2[4][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < kDig; i++)
#pragma unroll
      for (int j = 0; j < kDig; j++) {
        if (i + j >= kGroups) continue;
        if (i < j) {
          mma_f16(acc[0][i + j], A[i][0], A[i][1], A[i][2], A[i][3], A[j][0], A[j][2]);
          if (PAIR) mma_f16(acc[1][i + j], A[i][0], A[i][1], A[i][2], A[i][3], A[j][1], A[j][3]);
        } else if (i == j) {
          const __half2 half = __floats2half2_rn(0.5f, 0.5f);
          mma_f16(acc[0][i + j], A[i][0], A[i][1], A[i][2], A[i][3], h2_bits(__hmul2(bits_h2(A[i][0]), half)),
                  h2_bits(__hmul2(bits_h2(A[i][2]), half)));
          if (PAIR)
            mma_f16(acc[1][i + j], A[i][0], A[i][1], A[i][2], A[i][3], h2_bits(__hmul2(bits_h2(A[i][1]), half)),
                    h2_bits(__hmul2(bits_h2(A[i][3]), half)));
        }
        if (BLOCK1 && !PAIR) mma_f16(acc[1][i + j], A[i][0], A[i][1], A[i][2], A[i][3], B1[j][0], B1[j][1]);
        if (j < 4) mma_f16(acc[2][i + j], A[i][0], A[i][1], A[i][2], A[i][3], B2[j][0], B2[j][1]);
      }
  }
  // the diagonal's squares of d1 (G_2) and d2 (G_4), less their expectation
#pragma unroll
  for (int s = 2; s <= 4; s += 2) {
    acc[0][s][0] -= (g == 2 * q) ? diag0 : 0.f;
    acc[0][s][1] -= (g == 2 * q + 1) ? diag0 : 0.f;
    if (BLOCK1) {
      acc[1][s][2] -= (g == 2 * q) ? diag1 : 0.f;
      acc[1][s][3] -= (g == 2 * q + 1) ? diag1 : 0.f;
    }
  }
}

// One unit of a request (see accum_unit): its moment records into a.mom.  False, and
// nothing written, for a pair of which one run's walk has passed the limit: where chunks
// end shows in a run's last bits, which must not depend on the run it is paired with.
template <int DIM, bool PACK>
__device__ __forceinline__ bool digit_unit(const jne_accum_args& a, int unit, DigSmem& sm, const jne_round_keys& rk,
                                           int lane) {
  constexpr int d = DIM;
  constexpr bool PAIR = Packing<DIM, PACK>::kPair;
  constexpr bool BLOCK1 = PAIR || DIM > 8;
  constexpr int NU = Packing<DIM, PACK>::kRuns;
  constexpr int NQ = (d + 3) / 4;
  constexpr int NMWW = d * (d + 1) / 2, NMW = 3 * d, NNZW = d * d;
  constexpr int NREC = NMWW + NMW + NNZW + 3 * d;
  static_assert(NU * NREC <= kRecMax, "records of a unit fit the shared record");
  const int g = lane >> 2, q = lane & 3;
  const int run0 = NU * unit;
  const int nrun = min(NU, a.n_runs - run0);

  for (int e = lane; e < 16 * kZS; e += 32) {  // staging rows without a feature stay zero
    const int row = e / kZS;
    if ((PAIR ? (row & 7) : row) >= d) (&sm.zs[0][0])[e] = 0.f;
  }
  for (int e = lane; e < NMWW; e += 32) {
    int t = e, aa = 0;
    while (t >= d - aa) { t -= d - aa; aa++; }
    sm.mww_pr[e] = (unsigned short)(aa | ((aa + t) << 8));
  }
  const int rowA = g, rowB = PAIR ? g : g + 8;
  const int selA = rowA >= d && rowA < d + 4 ? rowA - d + 1 : 0;
  const int selB = rowB >= d && rowB < d + 4 ? rowB - d + 1 : 0;
  if (lane < 16) {
    sm.basis[0][lane] = 0u;
    sm.basis[1][lane] = 0x3C003C00u;  // 1, 1
    sm.wc[lane] = 0.0;
  }
  for (int e = lane; e < NU * NREC; e += 32) sm.rec[e] = 0.0;
  const int T = a.steps;
  const int L = jne_digit_chunk(T), sh = jne_digit_shift(T), limit = jne_digit_limit(T) << 8;
  const int h = L >> 1;
  // walk rows: units of 2^-(40 + sh); block 1's increment columns: digits from 2^-8 down, as block 2's
  const FixedScale scaleA = fixed_scale(40 + sh, 0);
  const FixedScale scaleB = PAIR || g < 4 ? scaleA : fixed_scale(42, 6);
  // expected squares of a tile on the diagonal (halved where the block holds half of i = j); the walk rows of
  // block 1 are its lanes g < 4
  const float diag0 = 0.5f * kSquareMean, diag1 = g < 4 ? (PAIR ? 0.5f * kSquareMean : kSquareMean) : 0.f;
  const uint32_t seed0 = a.seed_first + (uint32_t)run0;
  __syncwarp();

  for (int c0 = 0; c0 < T;) {
    float acc[3][kGroups][4];
#pragma unroll
    for (int n = 0; n < 3; n++)
#pragma unroll
      for (int s = 0; s < kGroups; s++)
#pragma unroll
        for (int r = 0; r < 4; r++) acc[n][s][r] = 0.f;
    long long carA = 0, carB = 0;
    int t0 = c0, over = 0;
    for (;;) {
      const int i = t0 + lane;
      const bool valid = i < T;
#pragma unroll
      for (int r = 0; r < NU; r++) {
        const int row0 = 8 * r;
#pragma unroll
        for (int j = 0; j < NQ; j++) {
          float z[4];
          jne_normal_quad((uint32_t)(i + 1), (uint32_t)j, seed0 + (uint32_t)r, rk, z);
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (4 * j + e < d) sm.zs[row0 + 4 * j + e][lane] = z[e];
        }
        if (!valid)
#pragma unroll
          for (int f = 0; f < d; f++) sm.zs[row0 + f][lane] = 0.f;
      }
      if (lane < 16) {  // the basis at steps 2 lane, 2 lane + 1: c and c^2 = 1024 eA + eB, |eB| <= 512
        const int ca = t0 - c0 + 2 * lane - h, cb = ca + 1;
        const int ea = (ca * ca + 512) >> 10, eb = (cb * cb + 512) >> 10;
        sm.basis[2][lane] = h2_bits(__floats2half2_rn((float)ca, (float)cb));
        sm.basis[3][lane] = h2_bits(__floats2half2_rn((float)ea, (float)eb));
        sm.basis[4][lane] = h2_bits(__floats2half2_rn((float)(ca * ca - 1024 * ea), (float)(cb * cb - 1024 * eb)));
      }
      __syncwarp();
      const int nvalid = min(32, T - t0);
      if (nvalid == 32)
        digit_tile<DIM, true, PACK>(sm.zs, sm.basis, g, q, nvalid, selA, selB, scaleA, scaleB, carA, carB, diag0, diag1,
                                    acc);
      else
        digit_tile<DIM, false, PACK>(sm.zs, sm.basis, g, q, nvalid, selA, selB, scaleA, scaleB, carA, carB, diag0,
                                     diag1, acc);
      __syncwarp();
      t0 += 32;
      if (PAIR) over = max(over, max(abs((int)(carA >> 32)), abs((int)(carB >> 32))));
      if (t0 >= T || t0 - c0 >= L) break;
      if (!PAIR) {
        const int hA = abs((int)(carA >> 32)), hB = BLOCK1 && g < 4 ? abs((int)(carB >> 32)) : 0;
        if (__any_sync(0xffffffffu, max(hA, hB) > limit)) break;
      }
    }
    if (PAIR && __any_sync(0xffffffffu, over > limit)) return false;
    const int Lc = min(t0, T) - c0;
    const int ntile = (t0 - c0) >> 5;
    // the squares of d3 left out with G_6 have a mean too, (1024^2 - 1) / 12 for every step but the chunk's first
    // (b = 0): 256/3 in units of G_5.
    const int left_out = ((Lc - 1) * 256 + 1) / 3;

    // ---- chunk end: the local Gram, staged in FP64 (cm[row][col], as in the mixed kernel: col < 16 walk columns,
    //      16 + f increments).  Symmetric blocks are staged doubled, their transposes added by the merge. ----
#pragma unroll
    for (int n = 0; n < 3; n++) {
      if (n == 1 && !BLOCK1) continue;
      const bool sym = n == 0 || (n == 1 && PAIR);
      const float k2 = sym ? 2.f : 1.f;
      const float back = (n == 0 ? diag0 : n == 1 ? diag1 : 0.f) * (float)ntile;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        if (PAIR && ((n == 0 && r >= 2) || (n == 1 && r < 2))) continue;
        const int lrow = r < 2 ? rowA : rowB;  // the row within its run
        const bool dg = (n == 0 && r < 2) || (n == 1 && r >= 2) ? g == 2 * q + (r & 1) : false;
        const float bk = dg ? back : 0.f;
        // (accumulator + expectation) x k2 may pass 2^24: add as integers
        const int bki = (int)(bk * k2);
        const int g0 = (int)(acc[n][0][r] * k2), g1 = (int)(acc[n][1][r] * k2), g3 = (int)(acc[n][3][r] * k2);
        const int g2 = (int)(acc[n][2][r] * k2) + bki, g4 = (int)(acc[n][4][r] * k2) + bki;
        const int g5 = (int)(acc[n][5][r] * k2) + (bki ? left_out : 0);
        // a basis row of a symmetric block: its only digit meets every digit of the column, so G_0 (halved) counts twice
        const int m0 = sym && lrow >= d ? 2 : 1;
        const double v = combine(g0 * m0, g1, g2, g3, g4, g5);
        const int row = r < 2 ? g : g + 8, e = 2 * q + (r & 1);
        int col;
        if (n == 0 || (PAIR && n == 1)) col = e;
        else if (n == 1) col = e < 4 ? 8 + e : 20 + e;
        else if (PAIR) col = 16 + (e & 3);
        else col = 16 + e;
        if (PAIR && n == 2 && (e < 4) != (r < 2)) continue;  // run A's rows with run B's increments and vice versa
        sm.cm[row][col] = v;
      }
    }
    if (q == 0) {
      const double u = __hiloint2double((1023 - 40 - sh) << 20, 0);  // 2^-(40 + sh)
      if (g < d) sm.tz[g] = int_to_f64(carA) * u;
      if (PAIR ? g < d : (BLOCK1 && g + 8 < d)) sm.tz[g + 8] = int_to_f64(carB) * u;
    }
    __syncwarp();
    // ---- merge into the records in FP64: W = wc + b; steps i + 1 = K + c, K = c0 + 1 + h ----
    const double dl = (double)Lc, K = (double)c0 + (double)(1 + h);
    const int s1 = Lc * (Lc - 1) / 2 - h * Lc;  // sum of c
    const int s2 = (Lc - 1) * Lc * (2 * Lc - 1) / 6 - h * Lc * (Lc - 1) + h * h * Lc;  // sum of c^2
    // units of the staged sums: a walk digit's 2^-sh (times 2^-50, see combine), and a product of two
    const double ub = __hiloint2double((1023 - 50 - sh) << 20, 0), uww = __hiloint2double((1023 - 50 - 2 * sh) << 20, 0);
    const int lf = PAIR ? (lane & 7) : lane, lr0 = PAIR ? (lane & 8) : 0;
    const bool lane_feature = lane_feature_of<DIM, PACK>(lane);
    constexpr double uz = 0x1p-8;  // an increment digit's
    if (lane_feature) {
      const int f = lf, x = lane, rb = (PAIR ? lane >> 3 : 0) * NREC;
      const double hb = PAIR || f < 8 ? 0.5 * ub : ub;  // symmetric blocks are staged doubled
      const double w = sm.wc[x], tz = sm.tz[x];
      const double Sb = sm.cm[lr0 + d][f] * hb, Scb = sm.cm[lr0 + d + 1][f] * hb;
      const double Seb = fma(sm.cm[lr0 + d + 2][f], 1024.0, sm.cm[lr0 + d + 3][f]) * hb;
      const double z1 = uz * 0x1p-50, Scz = sm.cm[lr0 + d + 1][16 + f] * z1;
      const double Sez = fma(sm.cm[lr0 + d + 2][16 + f], 1024.0, sm.cm[lr0 + d + 3][16 + f]) * z1;
      const double S1 = fma(dl, w, Sb);                       // sum W
      const double Sc = fma((double)s1, w, Scb);              // sum c W
      const double Se = fma((double)s2, w, Seb);              // sum c^2 W
      sm.sb[x] = Sb;
      sm.sw[x] = S1;
      double* rec = sm.rec + rb + NMWW;
      rec[f] += S1;
      rec[d + f] += fma(K, S1, Sc);
      rec[2 * d + f] += fma(K, fma(K, S1, 2.0 * Sc), Se);
      double* rz = sm.rec + rb + NMWW + NMW + NNZW + d;
      rz[f] += fma(K, tz, Scz);
      rz[d + f] += fma(K, fma(K, tz, 2.0 * Scz), Sez);
    }
    __syncwarp();
    for_slots<NU * NMWW, true>(lane, [&](int t) {
      const int r = NU == 1 ? 0 : t / NMWW, e = t - r * NMWW, o = 8 * r;
      const int p = sm.mww_pr[e] & 0xff, c = sm.mww_pr[e] >> 8;  // p <= c
      const double S = PAIR || c < 8 ? 0.5 * (sm.cm[o + p][c] + sm.cm[o + c][p]) : sm.cm[p][c];
      // sum (wp + bp)(wc + bc) = wc sum Wp + wp sum bc + sum bp bc
      sm.rec[r * NREC + e] += fma(sm.wc[o + c], sm.sw[o + p], fma(sm.wc[o + p], sm.sb[o + c], S * uww));
    });
    for_slots<NU * NNZW, true>(lane, [&](int t) {
      const int r = NU == 1 ? 0 : t / NNZW, tt = t - r * NNZW, za = tt / d, wb = tt - za * d, o = 8 * r;
      sm.rec[r * NREC + NMWW + NMW + tt] +=
          fma(sm.tz[o + za], sm.wc[o + wb], sm.cm[o + wb][16 + za] * (ub * uz));
    });
    __syncwarp();
    if (lane_feature) sm.wc[lane] += sm.tz[lane];
    __syncwarp();
    c0 = t0;
  }

  // ---- the records: y = (i + 1) / T ----
  if (lane_feature_of<DIM, PACK>(lane)) {
    const int r = PAIR ? lane >> 3 : 0, f = PAIR ? (lane & 7) : lane;
    double* rec = sm.rec + r * NREC;
    const double iT = 1.0 / (double)T;
    rec[jne_slot_MWy(f, d)] *= iT;
    rec[jne_slot_MWyy(f, d)] *= iT * iT;
    rec[jne_slot_Nzy(f, d)] *= iT;
    rec[jne_slot_Nzyy(f, d)] *= iT * iT;
    rec[jne_slot_Nz1(f, d)] = sm.wc[lane];
  }
  __syncwarp();
  const size_t ld = (size_t)a.mom_ld;
  for (int t = lane; t < NU * NREC; t += 32) {
    const int r = t / NREC, e = t - r * NREC;
    if (r < nrun) a.mom[(size_t)e * ld + run0 + r] = sm.rec[t];
  }
  __syncwarp();
  return true;
}

// The runs of a pair by themselves, as the unpacked kernel computes them (a walk passes the limit with
// probability 2e-11 per feature and chunk).  A call, and a check once a chunk, so that neither its registers
// nor its code touch the packed kernel's loop: ending the pair's chunk there and starting over with one run's
// chunks cost 3 - 4 % at dims 1 to 4, T 1000; this form -0.5 % at dims 1, 2 and 4, +2 % at dim 3 (T 10^4: -7 %).
template <int DIM>
__device__ __noinline__ void digit_pair_apart(const jne_accum_args& a, int unit, DigSmem& sm, const jne_round_keys& rk,
                                              int lane) {
  __syncwarp();
  for (int run = 2 * unit; run < min(2 * unit + 2, a.n_runs); run++) digit_unit<DIM, false>(a, run, sm, rk, lane);
}

template <int DIM, bool PACK>
__global__ void __launch_bounds__(kMixWarps * JNE_WARP, 3)
    k_accum_digits(const __grid_constant__ jne_accum_args a, const __grid_constant__ jne_round_keys rk,
                   const __grid_constant__ jne_finalize_args fin) {
  __shared__ DigSmem sm_all[kMixWarps];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nwarps = gridDim.x * kMixWarps;
  const bool fused = fin.out != nullptr && a.batch_done != nullptr;
  const long long units = jne_units(DIM, a.n_runs, PACK);
  // first unit by warp index, then the next free one from the counter
  for (long long unit = blockIdx.x * kMixWarps + wib; unit < units;) {
    const bool written = digit_unit<DIM, PACK>(a, (int)unit, sm_all[wib], rk, lane);
    if constexpr (Packing<DIM, PACK>::kPair)
      if (!written) digit_pair_apart<DIM>(a, (int)unit, sm_all[wib], rk, lane);
    if (fused) {
      const long long first = batch_complete(a.batch_done, unit, units, lane);
      if (first >= 0) finalize_batch(fin, first, PACK, lane);
      __syncwarp();
    }
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(a.next_run, 1ull);
    unit = nwarps + (long long)__shfl_sync(0xffffffffu, item, 0);
  }
}

template <int DIM>
cudaError_t launch_digits_dim(const jne_accum_args& a, const jne_finalize_args& fin, int sms, cudaStream_t st) {
  const int threads = kMixWarps * JNE_WARP;
  const bool pack = DIM <= JNE_PACK_MAX_DIM && jne_digits_pack(DIM, a.steps, a.n_runs, sms);
  auto k = pack ? k_accum_digits<DIM, (DIM <= JNE_PACK_MAX_DIM)> : k_accum_digits<DIM, false>;
  k<<<resident_grid(k, threads, 0, sms, jne_units(DIM, a.n_runs, pack), kMixWarps), threads, 0, st>>>(
      a, jne_make_round_keys(a.key0, a.key1), fin);
  return cudaGetLastError();
}

}  // namespace
