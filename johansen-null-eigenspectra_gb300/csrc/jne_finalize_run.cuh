// jne_finalize_run.cuh -- the per-run FP64 finalize (moment record -> eigenvalues),
// shared by the finalize kernels and by the mixed accumulation kernel, which
// finalizes its own runs in batches of 32 (one run per lane).
//
// Replaces johansen_statistics.rs:24-47 (the F-based Grams, then
// GeneralizedEigen(S10'S10, S11) via LAPACK dggev, |alpha|/beta, descending
// sort).  One thread per run, all in FP64:
//   1. F_j = G[x_j] - alpha_j * 1 - beta_j * (y - ybar) for the model's rows,
//      where G = [W; 1; y; y^2].  This is construct_f_matrix (:102-197) written as
//      a linear map: demeaning (models 2, 3) subtracts the row mean, model 4
//      subtracts the least-squares fit on {1, y}, here on the orthogonal pair
//      {1, y - ybar}.  A residual is orthogonal to what was subtracted, so
//      F_j F_l' = F_j G_l' needs one side's correction.
//      The walk stays unscaled: scaling a row of F does not change the pencil's
//      eigenvalues, and the factors dt of S11 and s^2 of S10'S10 (dB = s z) are
//      one factor of the result (lam_scale).
//   2. S11 = L L' (Cholesky, reciprocal pivots only), E = S10 L^-T, C = E'E: the
//      pencil's eigenvalues are those of the symmetric PSD matrix C.
//   3. Householder tridiagonalisation of one triangle + implicit QL (eigenvalues
//      only), then |lambda| and a descending sort -- the reference reports
//      |alpha|/beta.
// What bounds it: FP64 instructions.  On this GPU one warp's FP64 instruction
// holds its scheduler's FP64 pipe for 64 cycles (76 with all four busy), however
// many of its lanes are active, and dependent ones follow each other as fast as
// independent ones; so a warp finalizes 32 runs, one per lane, and the time is the
// instruction count.  At k = 13 about 7,500 are left of 12,000: the one-sided
// corrections and the unscaled walk (S, S10), rsqrt for sqrt and division, half the
// rank-two updates, the shift's correction in FP32 (any shift is a valid one: only
// the convergence depends on it) and the deflation test on exponents.
// Measured, whole calls: five models of 40,000 runs at dim 12, T 2000 (one launch for
// all models included) 11.25 -> 7.70 ms, 6.9 with QL's sweeps in one loop and 6.63 with
// two rows of E at a time; 20,011 runs at dim 6, T 100, mostly finalize, 765 -> 413 us.
// Errors against quad precision are no larger (dim 12, T 100, model 4: 4.1e-14 ->
// 2.3e-14 rms).
#pragma once
#include <cfloat>
#include <math_constants.h>
#include "jne_kernels.h"

namespace jne_fin {
namespace {  // internal linkage: each translation unit that includes this has its own copy

// The run's moment record, in units of the unscaled walk.
struct Ctx {
  const double* mom;
  long long ld;
  int run, d;
  const double* Y;
  // cached in L2 only: the mixed kernel reads records its own warp wrote moments earlier
  __device__ double rec(int slot) const { return __ldcg(mom + (size_t)slot * ld + run); }
  // M(r, n) = sum_i G_r G_n over the global basis G = [W (d); 1; y; y^2], r <= n
  __device__ double M(int r, int n) const {
    if (n < d) return rec(jne_slot_MWW(r, n, d));
    if (r < d) {
      const int p = n - d;
      return rec(p == 0 ? jne_slot_MW1(r, d) : p == 1 ? jne_slot_MWy(r, d) : jne_slot_MWyy(r, d));
    }
    return Y[(r - d) + (n - d)];
  }
  // N(r, c) = sum_i G_r z_c
  __device__ double N(int r, int c) const {
    if (r < d) return rec(jne_slot_NzW(c, r, d));
    const int p = r - d;
    return rec(p == 0 ? jne_slot_Nz1(c, d) : p == 1 ? jne_slot_Nzy(c, d) : jne_slot_Nzyy(c, d));
  }
};

// Householder reduction of a symmetric n x n matrix to tridiagonal form (Golub &
// Van Loan, Matrix Computations, Algorithm 8.3.1), given and overwritten as its
// strict upper triangle (A[i][j], i < j) and diagonal: diagonal -> dg[0..n-1],
// sub-diagonal -> eo[0..n-2].
__device__ __forceinline__ void tridiagonalize(double (*A)[JNE_MAX_K], int n, double* dg, double* eo) {
  for (int k = 0; k + 2 < n; k++) {
    double sigma = 0.0;
    for (int i = k + 2; i < n; i++) sigma = fma(A[k][i], A[k][i], sigma);
    const double x0 = A[k][k + 1];
    if (sigma == 0.0) { eo[k] = x0; continue; }
    const double r2 = fma(x0, x0, sigma);
    const double nrm = r2 * rsqrt(r2);
    const double alpha = x0 > 0.0 ? -nrm : nrm;  // H x = alpha e1
    double v[JNE_MAX_K], p[JNE_MAX_K];
    v[k + 1] = x0 - alpha;                        // |x0| + nrm: no cancellation
    for (int i = k + 2; i < n; i++) v[i] = A[k][i];
    const double tau = 1.0 / fma(nrm, fabs(x0), r2);  // 2 / (v'v)
    for (int i = k + 1; i < n; i++) p[i] = dg[i] * v[i];
    for (int i = k + 1; i < n; i++) {
      const double vi = v[i];
      double t = p[i];
      for (int j = i + 1; j < n; j++) {
        const double a = A[i][j];
        t = fma(a, v[j], t);
        p[j] = fma(a, vi, p[j]);
      }
      p[i] = t;
    }
    double pv = 0.0;
    for (int i = k + 1; i < n; i++) {
      p[i] *= tau;
      pv = fma(p[i], v[i], pv);
    }
    const double K = 0.5 * tau * pv;
    for (int i = k + 1; i < n; i++) p[i] = fma(-K, v[i], p[i]);  // w = p - K v
    for (int i = k + 1; i < n; i++) {
      const double vi = v[i], wi = p[i];
      dg[i] = fma(-2.0 * vi, wi, dg[i]);
      for (int j = i + 1; j < n; j++) A[i][j] = fma(-wi, v[j], fma(-vi, p[j], A[i][j]));
    }
    eo[k] = alpha;
  }
  if (n >= 2) eo[n - 2] = A[n - 2][n - 1];
}

// Biased exponent field of a double, as an integer to compare.
__device__ __forceinline__ int exponent_bits(double x) { return __double2hiint(x) & 0x7FF00000; }
__device__ __forceinline__ bool is_zero(double x) { return ((__double2hiint(x) & 0x7FFFFFFF) | __double2loint(x)) == 0; }

// Eigenvalues of the symmetric tridiagonal matrix (dg, eo) by the implicit QL
// method with Wilkinson shifts (Bowdler, Martin, Reinsch & Wilkinson, "The QR
// and QL algorithms for symmetric matrices", Numer. Math. 11, 1968).  eo[i]
// couples dg[i] and dg[i+1]; the sweep count per eigenvalue is bounded.  One loop
// over sweeps, whichever eigenvalue a lane is at: the warp then runs as many as its
// slowest lane in all, not the slowest lane's for each eigenvalue in turn.
__device__ __forceinline__ bool tridiagonal_ql(double* dg, double* eo, int n) {
  eo[n - 1] = 0.0;
  bool ok = true;
  int l = 0, sweeps = 0;
  for (;;) {
    int m = l;
    for (; l < n; l++, sweeps = 0) {
      // negligible by exponents, with no FP64 instruction: |eo| < eps max(|dg[m]|, |dg[m + 1]|) when it
      // breaks, within a factor of four of |eo| <= eps (|dg[m]| + |dg[m + 1]|); never for a NaN eo
      int em = exponent_bits(dg[l]);
      for (m = l; m < n - 1; m++) {
        const int en = exponent_bits(dg[m + 1]);
        if (exponent_bits(eo[m]) <= max(em, en) - (53 << 20) || is_zero(eo[m])) break;
        em = en;
      }
      if (m == l) continue;
      if (sweeps < 63) break;
      ok = false;  // not converged: on to the next eigenvalue
    }
    if (l >= n) return ok;
    sweeps++;
    // the shift d_l - e_l / (g + sign(g) sqrt(g^2 + 1)), g = (d_{l+1} - d_l) / (2 e_l): its correction in FP32
    const double dl = dg[l], el = eo[l];
    const float ef = (float)el, gf = (float)(dg[l + 1] - dl) / (2.0f * ef);
    double cf = (double)(ef / (gf + copysignf(sqrtf(fmaf(gf, gf, 1.0f)), gf)));
    if (!isfinite(cf)) {  // values outside FP32's range
      const double gd = (dg[l + 1] - dl) / (2.0 * el);
      cf = el / (gd + copysign(hypot(gd, 1.0), gd));
    }
    double d1 = dg[m];  // dg[i + 1]
    double g = d1 - dl + cf;
    double s = 1.0, c = 1.0, p = 0.0;
    int i = m - 1;
    for (; i >= l; i--) {
      const double e = eo[i], d0 = dg[i];
      const double f = s * e, b = c * e;
      // Givens rotation from one reciprocal square root (the moments keep
      // f and g far from the overflow / underflow range hypot guards)
      const double r2 = fma(f, f, g * g);
      if (is_zero(r2)) break;  // underflow
      const double ir = rsqrt(r2);
      eo[i + 1] = r2 * ir;
      s = f * ir;
      c = g * ir;
      g = d1 - p;
      const double r = fma(d0 - g, s, 2.0 * c * b);
      p = s * r;
      dg[i + 1] = g + p;
      g = fma(c, r, -b);
      d1 = d0;
    }
    if (i >= l) {  // recover from underflow
      eo[i + 1] = 0.0;
      dg[i + 1] = d1 - p;
    } else {
      dg[l] = d1 - p;
      eo[l] = g;
    }
    eo[m] = 0.0;
  }
}

// TWO: two rows of E at a time -- two independent chains of FP64 instructions for each
// element of L read, and one pass over C for both.  7% less time in the finalize
// kernel, where warps wait on the stack's loads (five models of 40,000 runs at k = 12,
// 13: 4.0 -> 3.7 ms); fused into an accumulation its code costs more than it saves
// (dim 12, T 1000: 5.57 -> 5.70 ms).  The same operations in the same order.
template <bool TWO>
__device__ __noinline__ void finalize_run(const jne_finalize_args& f, int run) {
  const int d = f.dim, model = f.model;
  const int k = (model == 1 || model == 3) ? d + 1 : d;
  const Ctx c{f.mom, f.mom_ld, run, d, f.ts.Y};
  const double T = (double)f.steps;
  const int ONE = d, Yr = d + 1, YY = d + 2;
  const int nb = (model == 2 || model == 4) ? d - 1 : d;    // walk rows kept
  const int last = model == 1 ? ONE : model == 4 ? YY : Yr;  // the row after them (none in model 0)
  const bool trend = model == 2 || model == 3;              // its row is y - 1/2
  const int proj = trend ? 1 : model == 4 ? 2 : 0;          // corrections: 1, or 1 and y

  // F rows: F_j = G[x_j] - al_j * 1 - be_j * (y - ybar)
  double al[JNE_MAX_K], be[JNE_MAX_K], m1[JNE_MAX_K], my[JNE_MAX_K];
  const double iT = 1.0 / T, ybar = f.ts.Y[1] * iT;
  if (proj >= 1)
    for (int j = 0; j < nb; j++) {
      m1[j] = c.M(j, ONE);
      al[j] = m1[j] * iT;  // row mean
    }
  if (trend) al[nb] = 0.5;
  if (proj == 2) {
    const double iS = 1.0 / f.ts.Syy;
    m1[nb] = f.ts.Y[2];
    al[nb] = m1[nb] * iT;
    for (int j = 0; j < k; j++) {
      my[j] = j < nb ? fma(-ybar, m1[j], c.M(j, Yr)) : f.ts.Syy2;  // sum (y - ybar) G_j
      be[j] = my[j] * iS;
    }
  }

  // S11 (lower triangle of S) and its Cholesky factor, row by row; inv[j] = 1 / L[j][j]
  double S[JNE_MAX_K][JNE_MAX_K];
  bool ok = true;
  double inv[JNE_MAX_K];
  for (int j = 0; j < k && ok; j++) {
    const int x = j < nb ? j : last;
    for (int i = 0; i <= j; i++) {
      double s;
      if (trend && j == nb) {
        // (y - 1/2) against the demeaned walk i (sum (y - 1/2) = 1/2), and against itself
        s = i < nb ? fma(-0.5, m1[i] + al[i], c.M(i, Yr)) : f.ts.Syh;
      } else if (proj == 2 && i == nb) {
        s = f.ts.Sr2;  // the residual of y^2
      } else {
        s = i < nb ? c.M(i, x) : c.M(x, x);
        if (proj >= 1) s = fma(-al[j], m1[i], s);
        if (proj == 2) s = fma(-be[j], my[i], s);
      }
      for (int p = 0; p < i; p++) s = fma(-S[j][p], S[i][p], s);
      if (i == j) {
        if (!(s > 0.0)) { ok = false; break; }
        inv[j] = rsqrt(s);
      } else {
        S[j][i] = s * inv[i];
      }
    }
  }
  double* out = f.out + (size_t)run * k;
  if (!ok) {
    for (int j = 0; j < k; j++) out[j] = CUDART_NAN;
    if (f.status) atomicOr(f.status, JNE_DEV_NOT_SPD);
    return;
  }
  // C = E'E with E = S10 L^-T, one row of E at a time: row cc solves
  // L e = S10[cc, :]' and adds e e' to C, so E is never stored.  C's strict
  // upper triangle lives in the upper triangle of S (L uses the lower one and
  // inv[] its diagonal), its diagonal in dg[].
  double dg[JNE_MAX_K], eo[JNE_MAX_K];
  for (int p = 0; p < k; p++) {
    dg[p] = 0.0;
    for (int q = p + 1; q < k; q++) S[p][q] = 0.0;
  }
  for (int cc = 0; cc < d; cc += TWO ? 2 : 1) {
    const bool two = TWO && cc + 1 < d;  // the last of an odd number of rows goes with a row of zeros
    const double n1 = proj >= 1 ? c.N(ONE, cc) : 0.0, ny = proj == 2 ? fma(-ybar, n1, c.N(Yr, cc)) : 0.0;
    const double n1b = two && proj >= 1 ? c.N(ONE, cc + 1) : 0.0;
    const double nyb = two && proj == 2 ? fma(-ybar, n1b, c.N(Yr, cc + 1)) : 0.0;
    double e[JNE_MAX_K], b[JNE_MAX_K];
    for (int j = 0; j < k; j++) {
      const int x = j < nb ? j : last;
      double s = c.N(x, cc), t = two ? c.N(x, cc + 1) : 0.0;
      if (proj >= 1) s = fma(-al[j], n1, s);
      if (proj == 2) s = fma(-be[j], ny, s);
      if (TWO) {
        if (proj >= 1) t = fma(-al[j], n1b, t);
        if (proj == 2) t = fma(-be[j], nyb, t);
      }
      for (int p = 0; p < j; p++) {
        const double l = S[j][p];
        s = fma(-l, e[p], s);
        if (TWO) t = fma(-l, b[p], t);
      }
      e[j] = s * inv[j];
      if (TWO) b[j] = t * inv[j];
    }
    for (int p = 0; p < k; p++) {
      const double ep = e[p], bp = TWO ? b[p] : 0.0;
      dg[p] = fma(ep, ep, dg[p]);
      if (TWO) dg[p] = fma(bp, bp, dg[p]);
      for (int q = 0; q < p; q++) {
        double v = fma(ep, e[q], S[q][p]);
        if (TWO) v = fma(bp, b[q], v);
        S[q][p] = v;
      }
    }
  }
  // The reductions square the entries of C.  Explicit increments in FP64 (the separate kernel, lam_scale = T) may put
  // them where squares overflow or lose bits, beyond 2^400 either way; its diagonal bounds a Gram matrix.  Then an exact
  // power of two takes C to 1 and the eigenvalues back.
  int top = 1023 << 20;
  if (TWO && f.lam_scale != 1.0) {
    top = 0;
    for (int p = 0; p < k; p++) top = max(top, exponent_bits(dg[p]));
  }
  const bool scaled = TWO && top != 0x7FF00000 && abs(top - (1023 << 20)) > (400 << 20);
  const int up = min(max((2046 << 20) - top, 1 << 20), 2045 << 20);  // the exponent field of 2^-e, for C of 2^e
  if (scaled) {
    const double to_one = __hiloint2double(up, 0);
    for (int p = 0; p < k; p++) {
      dg[p] *= to_one;
      for (int q = p + 1; q < k; q++) S[p][q] *= to_one;
    }
  }
  tridiagonalize(S, k, dg, eo);
  // (a single eigenvalue meets no sweep that a NaN or an infinity would keep from converging)
  const bool good = tridiagonal_ql(dg, eo, k) && !(k == 1 && exponent_bits(dg[0]) == 0x7FF00000);
  if (!good && f.status) atomicOr(f.status, JNE_DEV_NOT_SPD);
  for (int j = 0; j < k; j++) dg[j] = fabs(dg[j]) * f.lam_scale;
  if (scaled) {
    const double back = __hiloint2double((2046 << 20) - up, 0);
    for (int j = 0; j < k; j++) dg[j] *= back;
  }
  for (int j = 1; j < k; j++) {  // insertion sort, descending
    const double v = dg[j];
    int i = j - 1;
    while (i >= 0 && dg[i] < v) { dg[i + 1] = dg[i]; i--; }
    dg[i + 1] = v;
  }
  for (int j = 0; j < k; j++) out[j] = dg[j];
}

}  // namespace
}  // namespace jne_fin
