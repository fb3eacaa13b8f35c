#include "planner.h"

#include <algorithm>
#include <functional>
#include <queue>

namespace fqla_host {

int64_t makespan(std::vector<int64_t> costs, int64_t copies, int64_t machines, int64_t give_up) {
  if (costs.empty()) return 0;
  std::sort(costs.begin(), costs.end(), std::greater<int64_t>());
  if ((int64_t)costs.size() * copies <= machines) return costs.front();
  int64_t total = 0;
  for (int64_t c : costs) total += c * copies;
  const int64_t at_least = std::max(costs.front(), (total + machines - 1) / machines);
  if (at_least > give_up) return at_least;
  // min-heap of the SMs' finish times
  std::vector<int64_t> load((size_t)machines, 0);
  std::priority_queue<int64_t, std::vector<int64_t>, std::greater<int64_t>> heap(
      std::greater<int64_t>(), std::move(load));
  int64_t longest = 0;
  for (int64_t c : costs)
    for (int64_t i = 0; i < copies; ++i) {
      const int64_t end = heap.top() + c;
      heap.pop();
      heap.push(end);
      longest = std::max(longest, end);
    }
  return longest;
}

std::optional<Split> split_sequences(const std::vector<int64_t>& bounds, int64_t heads, int64_t n_sm,
                                     int64_t min_chunks, int64_t slices, int64_t split_cost) {
  const size_t n = bounds.empty() ? 0 : bounds.size() - 1;
  std::vector<int64_t> chunks(n);
  int64_t longest = 0;
  for (size_t i = 0; i < n; ++i) {
    chunks[i] = (bounds[i + 1] - bounds[i] + CHUNK - 1) / CHUNK;
    longest = std::max(longest, chunks[i]);
  }
  if (longest < 2 * min_chunks) return std::nullopt;
  const int64_t copies = heads * slices;

  std::vector<int64_t> costs;
  auto layout_cost = [&](int64_t limit, int64_t give_up) {
    costs.clear();
    for (int64_t c : chunks) {
      const int64_t parts = std::max<int64_t>(1, (c + limit - 1) / limit);
      const int64_t per = (c + parts - 1) / parts;
      for (int64_t i = 0; i < parts; ++i) {
        const int64_t seg = std::min(per, c - i * per);
        if (seg > 0) costs.push_back(seg + CTA_START_CHUNKS + (i ? SEGMENT_OVERHEAD_CHUNKS : 0));
      }
    }
    return makespan(costs, copies, n_sm, give_up);
  };

  const int64_t unsplit = layout_cost(longest, INT64_MAX);
  int64_t cheapest = INT64_MAX, last = longest;
  std::vector<std::pair<int64_t, int64_t>> cands;  // (limit, cost), coarsest first
  for (int64_t p = 2; p <= longest / min_chunks; ++p) {
    const int64_t limit = (longest + p - 1) / p;
    if (limit < min_chunks) break;
    if (limit == last) continue;
    last = limit;
    // a split more than 3 % above the cheapest so far can neither be the cheapest nor be chosen
    const int64_t give_up = cheapest == INT64_MAX ? INT64_MAX : cheapest * 103 / 100;
    const int64_t cost = layout_cost(limit, give_up);
    cands.emplace_back(limit, cost);
    cheapest = std::min(cheapest, cost);
  }
  if (cands.empty() || (double)(cheapest + split_cost) > 0.97 * (double)unsplit) return std::nullopt;
  int64_t limit = 0;
  for (auto& c : cands)
    if ((double)c.second <= 1.03 * (double)cheapest) {
      limit = c.first;
      break;
    }
  Split s;
  for (size_t r = 0; r < n; ++r) {
    s.seg_begin.push_back((int64_t)s.seg_bounds.size());
    const int64_t parts = std::max<int64_t>(1, (chunks[r] + limit - 1) / limit);
    const int64_t per = (chunks[r] + parts - 1) / parts;
    for (int64_t i = 0; i < parts; ++i) s.seg_bounds.push_back(bounds[r] + i * per * CHUNK);
  }
  s.seg_begin.push_back((int64_t)s.seg_bounds.size());
  s.seg_bounds.push_back(bounds.back());
  return s;
}

}  // namespace fqla_host
