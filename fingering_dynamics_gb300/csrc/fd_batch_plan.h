// How many strips each member of a batch is cut into, plain C++ so that it can
// be checked without a GPU.
//
// The persistent grid takes tiles (a band's strip) from a counter, tallest first,
// so an iteration ends when the last CTA has finished its tiles.  A caller gives
// the tallest strip it wants; cutting every member into strips just that tall
// leaves a last round that is partly empty (2,064 tiles on 760 CTAs: three
// rounds, the third 70% full), and a small batch fewer tiles than CTAs (eight
// lattices of 256 x 512 in strips of 32 rows: 256 tiles).  So strips are cut
// shorter, the tallest first, while the tiles still fit the rounds, and the
// round count whose greedy schedule ends earliest is kept.  A strip costs its
// rows plus the time of about four (its first rows are loaded before the first
// one is computed).
#pragma once

#include <algorithm>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

namespace fd {

constexpr int kStripFill = 4;     // rows' time a strip's prologue costs
constexpr int kStripMinRows = 4;  // no strip is cut shorter
constexpr int kMaxPlanRounds = 16;  // beyond, the partly empty round is a small share

// heights and band counts of the members (0 bands: left out)
struct BatchShape {
  std::vector<int> height, bands;
};

inline int strip_rows(int height, int strips) { return (height + strips - 1) / strips; }

// Time (in rows) at which a greedy schedule, tallest strips first, ends on `grid` CTAs.
inline long long batch_makespan(const BatchShape& s, const std::vector<int>& strips, int grid) {
  std::vector<int> tiles;
  for (size_t i = 0; i < s.height.size(); ++i) {
    if (s.bands[i] == 0) continue;
    const int r = strip_rows(s.height[i], strips[i]);
    for (int y = 0; y < s.height[i]; y += r)
      tiles.insert(tiles.end(), (size_t)s.bands[i], std::min(r, s.height[i] - y) + kStripFill);
  }
  std::sort(tiles.begin(), tiles.end(), std::greater<int>());
  std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free;
  for (int g = 0; g < grid; ++g) free.push(0);
  long long end = 0;
  for (int t : tiles) {
    const long long at = free.top() + t;
    free.pop();
    free.push(at);
    end = std::max(end, at);
  }
  return end;
}

// Strips per member, each at most `rows` high.
inline std::vector<int> plan_strips(const BatchShape& s, int rows, int grid) {
  const size_t n = s.height.size();
  std::vector<int> base(n);
  long long tiles = 0;
  for (size_t i = 0; i < n; ++i) {
    base[i] = (s.height[i] + rows - 1) / rows;
    tiles += (long long)base[i] * s.bands[i];
  }
  if (grid < 1 || tiles == 0) return base;
  const long long first = (tiles + grid - 1) / grid;
  if (first > kMaxPlanRounds) return base;
  std::vector<int> best = base;
  long long best_end = batch_makespan(s, base, grid);
  for (long long rounds = first; rounds < first + 4; ++rounds) {
    std::vector<int> strips = base;
    long long left = rounds * grid - tiles;
    std::priority_queue<std::pair<int, int>> tallest;  // (rows, member)
    for (size_t i = 0; i < n; ++i)
      if (s.bands[i] > 0) tallest.push({strip_rows(s.height[i], strips[i]), (int)i});
    while (!tallest.empty()) {
      const int i = tallest.top().second;
      tallest.pop();
      if (s.bands[i] > left || strip_rows(s.height[i], strips[i] + 1) < kStripMinRows) continue;
      left -= s.bands[i];
      strips[i] += 1;
      tallest.push({strip_rows(s.height[i], strips[i]), i});
    }
    const long long end = batch_makespan(s, strips, grid);
    if (end < best_end) {
      best_end = end;
      best = strips;
    }
  }
  return best;
}

}  // namespace fd
