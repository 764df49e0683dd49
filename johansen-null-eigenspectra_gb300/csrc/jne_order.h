// jne_order.h -- the order in which warps take the units of a ragged launch
// (results do not depend on it).  Host code only.
#pragma once
#include <algorithm>
#include <numeric>
#include <tuple>
#include <vector>

namespace jne_detail {

// One piece of a launch: its request's dim, eigenvalue count and steps, and its units.
struct OrderItem {
  int dim, k, steps;
  long long units;
};

// Large dims first, so that the launch ends on short solves (a batch's solve takes
// 0.5 ms at k = 13, and nothing hides the last one's) and warps of an SM run the same
// dim's code; within a dim the longest paths first.  The 60-pair plan (128,000 runs)
// 15.4 -> 12.9 ms; batches of 25 to 60 requests of tens to hundreds of runs 2.0 - 3.3 ->
// 1.0 - 1.5 ms (longest paths first whatever the dim: 14.3 and 1.7 - 2.7).
//
// That order leaves few long paths of a small dim to the end, where they run alone.  So
// a piece at least eight times as long as the launch's mean unit, whose last unit, started
// in its turn, would end an eighth after both the time all warps need together and the
// longest unit, goes to the front, longest first.  100,000 runs at dim 12, T 1000 and 64
// at dim 1, T 10^5: 7.25 -> 5.98 ms; three models of dim 8, T 2000 and 200 runs at dim 2,
// T 5 10^4: 3.87 -> 3.13.  Shorter paths stay in turn: without the eight, batches of T
// 1000 to 10,000 mixed dims at their front and took up to 1.4 times as long (four: 1.06).
// Times are in 32-step tiles, which cost about the same at every dim (1.5 - 1.8 us a
// warp; a unit is a pair of runs at dims 1 to 4), and the solve that follows a batch's
// last unit, about k^3 / 7 of them.
inline std::vector<int> launch_order(const std::vector<OrderItem>& items, long long warps) {
  std::vector<int> order(items.size());
  std::iota(order.begin(), order.end(), 0);
  auto key = [&](int i) { return std::make_tuple(-items[i].dim, -items[i].k, -items[i].steps); };
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return key(x) < key(y); });
  auto tiles = [&](int i) { return (double)(items[i].steps / 32 + (items[i].steps % 32 != 0)); };
  auto length = [&](int i) { return tiles(i) + (double)items[i].k * items[i].k * items[i].k / 7.0; };
  double all = 0.0, longest = 0.0;
  long long n = 0;
  for (int i : order) {
    all += (double)items[i].units * tiles(i);
    n += items[i].units;
    longest = std::max(longest, length(i));
  }
  const double limit = 1.125 * std::max(all / (double)warps, longest);
  const double is_long = n > 0 ? 8.0 * all / (double)n : 0.0;  // eight mean units
  std::vector<int> early;
  double early_work = 0.0;
  long long early_units = 0;
  for (int pass = 0; pass < 4; pass++) {  // what goes to the front delays the rest, so look again (once or twice)
    std::vector<int> rest;
    double work = early_work;
    long long units = early_units;
    for (int i : order) {
      work += (double)items[i].units * tiles(i);
      units += items[i].units;
      // the units dealt out at the start do not wait
      const double start = units > warps ? work / (double)warps : 0.0;
      (tiles(i) >= is_long && start + length(i) > limit ? early : rest).push_back(i);
    }
    if (rest.size() == order.size()) break;
    order.swap(rest);
    early_work = 0.0;
    early_units = 0;
    for (int i : early) {
      early_work += (double)items[i].units * tiles(i);
      early_units += items[i].units;
    }
  }
  std::stable_sort(early.begin(), early.end(), [&](int x, int y) { return length(x) > length(y); });
  early.insert(early.end(), order.begin(), order.end());
  return early;
}

}  // namespace jne_detail
