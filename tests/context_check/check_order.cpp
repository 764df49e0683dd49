// The order of a ragged launch's pieces, on a model of the launch (every warp takes the next unit when it is free,
// a tile costs one unit of time, and a solve of k^3 / 7 follows the last unit): no mix may take much longer than its work or its longest path needs, and where
// nothing runs late the order is by falling dim, eigenvalue count and steps.
#include <cstdio>
#include <functional>
#include <queue>
#include <random>

#include "../../johansen-null-eigenspectra_gb300/csrc/jne_order.h"

using jne_detail::OrderItem;

namespace {

int failures = 0;
void check(bool ok, const char* what, double x, double y) {
  if (!ok) {
    failures++;
    std::printf("FAILED: %s (%g, %g)\n", what, x, y);
  }
}

double tiles(const OrderItem& o) { return (o.steps + 31) / 32; }

double solve(const OrderItem& o) { return (double)o.k * o.k * o.k / 7.0; }

// When the last unit of the launch and its solve are done.
double makespan(const std::vector<OrderItem>& items, const std::vector<int>& order, int warps) {
  std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
  for (int w = 0; w < warps; w++) free_at.push(0.0);
  double end = 0.0;
  for (int i : order)
    for (long long u = 0; u < items[(size_t)i].units; u++) {
      const double t = free_at.top() + tiles(items[(size_t)i]);
      free_at.pop();
      free_at.push(t);
      end = std::max(end, t + solve(items[(size_t)i]));
    }
  return end;
}

double least(const std::vector<OrderItem>& items, int warps) {
  double all = 0.0, longest = 0.0;
  for (const OrderItem& o : items) {
    all += (double)o.units * tiles(o);
    longest = std::max(longest, tiles(o) + solve(o));
  }
  return std::max(all / warps, longest);
}

bool permutation_of_all(std::vector<int> order, size_t n) {
  std::sort(order.begin(), order.end());
  for (size_t i = 0; i < order.size(); i++)
    if (order[i] != (int)i) return false;
  return order.size() == n;
}

bool by_dim(const std::vector<OrderItem>& items, const std::vector<int>& order) {
  auto key = [&](int i) { return std::make_tuple(-items[(size_t)i].dim, -items[(size_t)i].k, -items[(size_t)i].steps); };
  for (size_t p = 1; p < order.size(); p++)
    if (key(order[p]) < key(order[p - 1])) return false;
  return true;
}

}  // namespace

int main() {
  const int warps = 2432;
  // few long paths of a small dim beside many short ones of a large dim, given first or last
  const std::vector<std::vector<OrderItem>> late = {
      {{1, 1, 100000, 32}, {12, 12, 1000, 100000}},
      {{12, 12, 1000, 100000}, {1, 1, 100000, 32}},
      {{2, 3, 50000, 100}, {8, 8, 2000, 20000}, {8, 9, 2000, 20000}, {8, 8, 2000, 20000}},
      {{12, 13, 500, 50000}, {3, 3, 20000, 500}, {5, 6, 300, 400}},
  };
  for (const auto& items : late) {
    const double t = makespan(items, jne_detail::launch_order(items, warps), warps), l = least(items, warps);
    check(t < 1.2 * l, "a long path left to the end", t, l);
  }
  // random mixes of a few long pieces and many short ones, against the longest paths first whatever the dim (the whole
  // multiples of a long path that a launch may need are in both)
  std::mt19937 rng(7);
  auto log_uniform = [&](double lo, double hi) {
    return (int)std::exp(std::uniform_real_distribution<>(std::log(lo), std::log(hi))(rng));
  };
  for (int t = 0; t < 200; t++) {
    std::vector<OrderItem> items;
    const int n_long = (int)(rng() % 4), n = n_long + 1 + (int)(rng() % 20);
    for (int i = 0; i < n; i++) {
      const int dim = 1 + (int)(rng() % 12), k = dim + (int)(rng() % 2);
      if (i < n_long) items.push_back({dim, k, log_uniform(20000, 100000), log_uniform(1, 100)});
      else items.push_back({dim, k, log_uniform(256, 1000), log_uniform(1000, 20000)});
    }
    std::shuffle(items.begin(), items.end(), rng);
    const std::vector<int> order = jne_detail::launch_order(items, warps);
    check(permutation_of_all(order, items.size()), "a permutation", t, n);
    std::vector<int> longest((size_t)n);
    for (int i = 0; i < n; i++) longest[(size_t)i] = i;
    std::stable_sort(longest.begin(), longest.end(),
                     [&](int x, int y) { return items[(size_t)x].steps > items[(size_t)y].steps; });
    const double m = makespan(items, order, warps), l = makespan(items, longest, warps);
    check(m < 1.3 * l, "a mix", m, l);
  }
  // the 60 pairs of models and dims: no path is long beside the launch
  std::vector<OrderItem> pairs;
  for (int m = 0; m < 5; m++)
    for (int d = 1; d <= 12; d++)
      pairs.push_back({d, m == 1 || m == 3 ? d + 1 : d, (m * 12 + d) % 3 == 0 ? 10000 : 1000, d <= 4 ? 1000 : 2000});
  check(by_dim(pairs, jne_detail::launch_order(pairs, warps)), "sixty pairs by dim", 0, 0);
  // a launch whose units all start at once, and the empty one
  check(by_dim(late[0], jne_detail::launch_order(late[0], 1 << 20)), "no unit waits", 0, 0);
  check(jne_detail::launch_order({}, warps).empty(), "no pieces", 0, 0);
  std::printf("%d failures\n", failures);
  return failures != 0;
}
