// Blocks per solve of a batch, by timing (host code only).
#pragma once
#include <algorithm>
#include <vector>

namespace e3d {

// n solves on `blocks` blocks, at most most_parts for one of them.  limit(j, k): the
// blocks that solve j can use of k; nodes(j): its nodes; time(plan, ms): milliseconds
// of some iterations of the batch with plan[j] blocks for solve j, returns a status;
// warm(plan): the shortest such run.
// The plan that took least goes to best_plan.
//
// The first run in a process takes longer (the driver sets the kernel's stack up), so
// one goes ahead of those that count: without it six solves of 64^3 got 64 blocks
// each, 80 ms a batch where 25 take 61.  A time that is not positive counts for
// nothing.
template <typename Limit, typename Nodes, typename Warm, typename Time>
int pick_parts(size_t n, int blocks, int most_parts, Limit&& limit, Nodes&& nodes, Warm&& warm, Time&& time,
               std::vector<int>& best_plan) {
  std::vector<std::vector<int>> plans;
  double best = 1e300, ms = 0.0;
  auto attempt = [&](auto&& k_of) -> int {
    std::vector<int> p(n);
    for (size_t j = 0; j < n; ++j) p[j] = limit(j, k_of(j));
    if (std::find(plans.begin(), plans.end(), p) != plans.end()) return 0;
    if (plans.empty())
      if (int rc = warm(p)) return rc;
    plans.push_back(p);
    if (int rc = time(p, &ms)) return rc;
    if (ms > 0.0 && ms < best) {
      best = ms;
      best_plan = p;
    }
    return 0;
  };
  // Many blocks first: where few solves leave most blocks idle, the long runs with
  // few of them are not made.
  for (int k = 64; k >= 1 && ms < 1.5 * best; k /= 2)
    if (int rc = attempt([&](size_t) { return k; })) return rc;
  // A few solves: an even share of the blocks each, beyond the powers of two that
  // are close together (25 blocks, not 16 or 32, for six solves).
  const int share = blocks / (int)n;
  if (share > 16)
    if (int rc = attempt([&](size_t) { return std::min(share, most_parts); })) return rc;
  for (int per : {16384, 32768, 65536, 131072}) {
    const int rc = attempt([&](size_t j) {
      int k = 1;
      while (k < 64 && (long long)per * k * 3 < nodes(j) * 2) k *= 2;  // nearest power of two
      return k;
    });
    if (rc) return rc;
  }
  return 0;
}

}  // namespace e3d
