// Placement of buffers with known lifetimes in one piece of memory: host logic only.
#pragma once
#include <stddef.h>

#include <algorithm>
#include <utility>
#include <vector>

namespace ac {

struct Slot {
  size_t bytes = 0;
  int first = 0, last = 0;       // steps that touch it, both included
  size_t offset = 0;
  size_t end() const { return offset + (bytes + 255) / 256 * 256; }
  bool meets(const Slot& o) const { return first <= o.last && o.first <= last; }
};

// First fit, the largest first: two slots share bytes only if their lifetimes are disjoint. `fixed` are in place already.
// Returns the bytes that the slots reach to.
inline size_t place_slots(std::vector<Slot>& slots, const std::vector<Slot>& fixed = {}) {
  std::vector<size_t> order(slots.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return slots[a].bytes > slots[b].bytes; });
  std::vector<Slot> placed = fixed;
  size_t top = 0;
  for (size_t i : order) {
    Slot& s = slots[i];
    std::vector<std::pair<size_t, size_t>> busy;
    for (const Slot& o : placed)
      if (s.meets(o)) busy.push_back({o.offset, o.end()});
    std::sort(busy.begin(), busy.end());
    s.offset = 0;
    for (auto& b : busy) {
      if (s.end() <= b.first) break;
      s.offset = std::max(s.offset, b.second);
    }
    top = std::max(top, s.end());
    placed.push_back(s);
  }
  return top;
}

}  // namespace ac
