// Share-out of elements and node copies over the blocks of the one-barrier step
// kernel (see local_plan.hpp).
#include "local_plan.hpp"

#include <algorithm>

namespace dl {

namespace {
constexpr int32_t kOwned = static_cast<int32_t>(0x80000000u);
constexpr int kDegrees = 64;  // nodes of more slots count as nodes of 63
}  // namespace

void share_nodes(const HostLattice &h, int chunk, int blocks, LocalShare &s) {
  s.chunk = chunk;
  s.blocks = blocks;
  s.cap = 0;
  s.ptr.assign(static_cast<size_t>(blocks) + 1, 0);
  s.nodes.clear();
  s.nodes.reserve(static_cast<size_t>(h.N) + h.N / 4);
  std::vector<int32_t> seen(h.N, -1);  // the last block that has the node
  for (int b = 0; b < blocks; ++b) {
    const size_t e1 = static_cast<size_t>(std::min<int64_t>(h.E, (static_cast<int64_t>(b) + 1) * chunk));
    for (size_t i = 2 * static_cast<size_t>(b) * chunk; i < 2 * e1; ++i) {
      const int32_t n = h.conn[i];
      if (seen[n] == b) continue;
      s.nodes.push_back(seen[n] < 0 ? n | kOwned : n);
      seen[n] = b;
    }
    s.ptr[b + 1] = static_cast<int32_t>(s.nodes.size());
    s.cap = std::max(s.cap, s.ptr[b + 1] - s.ptr[b]);
  }
}

void share_ends(const HostLattice &h, LocalShare &s) {
  s.ends.resize(h.E);
  std::vector<int32_t> at(h.N), run(s.cap);
  auto degree = [&](int32_t id) {
    const int32_t n = id & ~kOwned;
    return std::min(h.slot_ptr[n + 1] - h.slot_ptr[n], kDegrees - 1);
  };
  for (int b = 0; b < s.blocks; ++b) {
    int32_t *const first = s.nodes.data() + s.ptr[b];
    const int count = s.ptr[b + 1] - s.ptr[b];
    // counting sort, most slots first, else in the order they came in
    int start[kDegrees] = {}, where = 0;
    for (int i = 0; i < count; ++i) ++start[degree(first[i])];
    for (int d = kDegrees - 1; d >= 0; --d) {
      const int c = start[d];
      start[d] = where;
      where += c;
    }
    for (int i = 0; i < count; ++i) run[start[degree(first[i])]++] = first[i];
    for (int i = 0; i < count; ++i) {
      first[i] = run[i];
      at[run[i] & ~kOwned] = i;
    }
    const size_t e1 = static_cast<size_t>(std::min<int64_t>(h.E, (static_cast<int64_t>(b) + 1) * s.chunk));
    for (size_t e = static_cast<size_t>(b) * s.chunk; e < e1; ++e)
      s.ends[e] = static_cast<uint32_t>(at[h.conn[2 * e]]) | (static_cast<uint32_t>(at[h.conn[2 * e + 1]]) << 16);
  }
}

}  // namespace dl
