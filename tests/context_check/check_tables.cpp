// The tables a context keeps on the device (chunk times, FP64 entries) after a failed allocation or upload: the next
// request must upload its own table again, never launch on a freed buffer or on another request's values.
#include "fake_cuda.h"

#include <cstdio>

using namespace jne_detail;

int jne_eigen_count(int model, int dim) { return model == 1 || model == 3 ? dim + 1 : dim; }

// One entry per (model, dim), recognisable by its values.
int jne_build_f64_entries(int model, int d, int4* out, int) {
  out[0] = make_int4(model, d, 0, 0);
  return 1;
}

namespace {

int failures = 0;
void check(bool ok, const char* what) {
  if (!ok) {
    failures++;
    std::printf("FAILED: %s\n", what);
  }
}

struct Bench {
  jne_context c;
  std::vector<double> mom;
  Bench() : mom(16 * 294) {
    c.budget = 1ull << 30;
    c.sms = 1;
    cudaMalloc((void**)&c.d_status, 4);
    cudaMalloc((void**)&c.d_next_run, 8);
  }
  int mixed(int steps) { return accumulate(&c, 0, 2, steps, 1, 2, 1, 4, JNE_PREC_MIXED, nullptr, mom.data(), nullptr); }
  int increments(int model, int dim) {
    return accumulate(&c, model, dim, 100, 0, 0, 0, 4, JNE_PREC_FP64, mom.data(), mom.data(), nullptr);
  }
};

bool own_table(const fake::MixedLaunch& l) {
  std::vector<jne_chunk_time> want((l.a.steps + l.a.chunk - 1) / l.a.chunk);
  fill_chunk_table(l.a.steps, l.a.chunk, want.data());
  return l.table.size() == want.size() && !std::memcmp(l.table.data(), want.data(), want.size() * sizeof want[0]);
}

}  // namespace

int main() {
  {  // the chunk table's buffer is lost in a failed growth
    Bench b;
    check(b.mixed(256) == JNE_OK && own_table(fake::mixed.back()), "first table");
    fake::fail_malloc = true;
    check(b.mixed(4096) == JNE_ERR_CUDA, "a failed growth is reported");
    fake::fail_malloc = false;
    check(b.mixed(256) == JNE_OK && own_table(fake::mixed.back()), "the old request after a failed growth");
    check(b.mixed(4096) == JNE_OK && own_table(fake::mixed.back()), "the new request after a failed growth");
  }
  {  // the chunk table's upload fails: its contents are undefined
    Bench b;
    check(b.mixed(4096) == JNE_OK, "first table");
    fake::fail_upload = true;
    check(b.mixed(2048) == JNE_ERR_CUDA, "a failed upload is reported");
    fake::fail_upload = false;
    std::memset((void*)b.c.d_ctab, 0xFF, b.c.ctab_cap * sizeof(jne_chunk_time));
    check(b.mixed(4096) == JNE_OK && own_table(fake::mixed.back()), "the old request after a failed upload");
  }
  {  // the entry table, whose count is rewritten ahead of its upload
    Bench b;
    check(b.increments(1, 2) == JNE_OK && fake::entries.back().size() == 1, "first entries");
    fake::fail_upload = true;
    check(b.increments(0, 3) == JNE_ERR_CUDA, "a failed entry upload is reported");
    fake::fail_upload = false;
    std::memset((void*)b.c.d_ent, 0xFF, b.c.ent_cap * sizeof(int4));
    check(b.increments(1, 2) == JNE_OK && fake::entries.back()[0].x == 1 && fake::entries.back()[0].y == 2,
          "the old entries after a failed upload");
  }
  std::printf("%d failures\n", failures);
  return failures != 0;
}
