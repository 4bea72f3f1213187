// Which elements and node copies each block of the one-barrier step kernel
// (local.cuh) takes.  Host only.
#pragma once

#include <cstdint>
#include <vector>

#include "setup.hpp"

namespace dl {

struct LocalShare {
  int chunk = 0, blocks = 0;   // block b takes the elements [b chunk, (b + 1) chunk)
  int cap = 0;                 // most node copies of a block
  std::vector<int32_t> ptr;    // [blocks + 1] runs of nodes
  std::vector<int32_t> nodes;  // node, sign bit set where this block owns it
  std::vector<uint32_t> ends;  // [E] the two end nodes as copies of the element's block (16 bits each)
};

// The runs of nodes (ptr, nodes, cap): a block's nodes in the order in which its
// elements touch them, owned by the first block that does.
void share_nodes(const HostLattice &h, int chunk, int blocks, LocalShare &s);

// Sorts each run by the nodes' numbers of slots, so that most warps of the node
// phase sum runs of equal length, and fills `ends`.  Needs cap <= 0xffff.
void share_ends(const HostLattice &h, LocalShare &s);

}  // namespace dl
