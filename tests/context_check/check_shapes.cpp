// The launch shape a mixed request reaches its kernel with: the size rule by default, the caller's packing at every
// size, and what the tuner times and keeps on either side of the rule's line.
#include "fake_cuda.h"

#include <cstdio>

cudaError_t jne_launch_export(int, int, int, uint32_t, uint32_t, uint32_t, double, double*, uint32_t*, cudaStream_t) {
  return cudaSuccess;
}
int jne_build_f64_entries(int, int, int4*, int) { return 0; }

namespace {

int failures = 0;
void check(bool ok, const char* what, long long x = 0, long long y = 0) {
  if (!ok) {
    failures++;
    std::printf("FAILED: %s (%lld, %lld)\n", what, x, y);
  }
}

bool packed(jne_context* c, int dim, int64_t n, int steps = 1000) {
  std::vector<double> out((size_t)n * jne_eigen_count(0, dim));
  check(jne_eigs_seeded(c, 0, dim, steps, 1, 1, n, JNE_PREC_MIXED, out.data()) == JNE_OK, "request");
  return fake::mixed.back().a.pack >= 0;
}

}  // namespace

int main() {
  const int64_t line = 16 * fake::kSms;
  for (int dim = 1; dim <= JNE_PACK_MAX_DIM; dim++) {
    jne_context* c = nullptr;
    check(jne_open(0, 0, &c) == JNE_OK, "open");
    for (int64_t n : {(int64_t)1, line - 1, line, line + 1, 4 * line}) {
      check(packed(c, dim, n) == (n > line), "the size rule", dim, n);
      for (int bps : {4, 6})
        for (int pack : {1, 0}) {
          jne_context* d = nullptr;
          check(jne_open(0, 0, &d) == JNE_OK && jne_set_launch_shape(d, bps, pack) == JNE_OK, "shape");
          check(packed(d, dim, n) == (pack == 1), "the caller's packing", pack, n);
          check(fake::mixed.back().a.blocks_per_sm == bps, "the caller's blocks", bps, n);
          jne_close(d);
        }
    }
    for (int steps : {1000 * dim * dim, 1000 * dim * dim + 1, 50000})  // long paths: from 12 runs per SM on
      for (int64_t n : {12 * fake::kSms, 12 * fake::kSms + 1, 16 * fake::kSms + 1})
        check(packed(c, dim, n, steps) == (n > (steps > 1000 * dim * dim ? 12 : 16) * fake::kSms), "long paths", steps, n);
    // the tuner: each row times the packing it names; the stored shape leaves the other side of the line to the rule
    for (int64_t n : {line / 2, 8 * line})
      for (bool packed_faster : {false, true}) {
        fake::ms = [&](const fake::MixedLaunch& l) { return (l.a.pack >= 0) == packed_faster ? 1.0f : 2.0f; };
        jne_tune_entry table[64], best{};
        int rows = 0;
        check(jne_autotune(c, dim, 700, 1e-6, 4, n, table, 64, &rows, &best) == JNE_OK, "autotune");
        for (int r = 0; r < rows; r++)
          if (table[r].ms >= 0)
            check(table[r].ms == ((table[r].pack == 1) == packed_faster ? 1.0 : 2.0), "a row's own packing", dim, n);
        check((best.pack == 1) == packed_faster, "the faster packing is chosen", dim, n);
        jne_set_chunk(c, JNE_CHUNK_TUNED);
        check(packed(c, dim, n) == packed_faster, "the choice at the timed size", dim, n);
        const int64_t other = n > line ? line / 2 : 8 * line;
        const bool by_rule = packed_faster == (n > line);
        check(packed(c, dim, other) == (by_rule ? other > line : packed_faster), "the other side of the line", dim, n);
        jne_set_chunk(c, 0);
      }
    jne_close(c);
  }
  {  // the shape serves every model, so the tuner times the one that merges the most moments (every kind: model 4)
    jne_context* c = nullptr;
    check(jne_open(0, 0, &c) == JNE_OK, "open");
    jne_tune_entry table[64], best{};
    int rows = 0, timed = 0, launches = 0;
    fake::ms = nullptr;
    const size_t before = fake::mixed.size();
    check(jne_autotune(c, 3, 700, 1e-6, 4, 500, table, 64, &rows, &best) == JNE_OK, "autotune");
    for (int r = 0; r < rows; r++) timed += table[r].ms >= 0;
    for (size_t i = before; i < fake::mixed.size(); i++)
      if (fake::mixed[i].a.n_runs == 500) {
        launches++;
        check(fake::mixed[i].a.model == 4 && fake::mixed[i].fin_model == 4, "the timed model", fake::mixed[i].a.model);
      }
    check(timed > 0 && launches == 3 * timed, "three launches a row", timed, launches);
    jne_close(c);
  }
  std::printf("%d failures\n", failures);
  return failures != 0;
}
