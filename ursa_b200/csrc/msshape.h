// msshape.h -- the grid of the many-source BFS (msbfs.cu).  Host code only, so
// that it can be checked without a GPU.
//
// A level of a small graph is too little work for the grid: on R-MAT-16 78%
// of the warps' time was the wait at the level's barrier.  So the grid is cut
// into groups of blocks, each with its own barrier and masks and every
// groups-th batch: while one group waits, another one's blocks work.  R-MAT-16
// from every node with 1 / 6 / 16 / 32 / 64 groups: 89.6 / 46.0 / 34.4 / 27.3 /
// 20.7 ms; 64 is what a block's share of nodes and the masks' memory allow there.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace ug {

constexpr uint64_t kMsGroups = 128;          // at most
constexpr uint64_t kMsNodesPerBlock = 8192;  // at most, of a group's pass
constexpr uint64_t kMsMaskBytes = 512ull << 20;  // of all groups
constexpr uint64_t kMsBlockNodes = 256;      // a warp per 32 nodes is all a level pass uses

struct MsShape {
  uint32_t groups, group_blocks;
};

// Groups and blocks per group for n >= 1 nodes, n_sources >= 1 in batches of
// 64 * W, and `resident` blocks that run at the same time (the blocks of a
// group wait for one another, so there are never more).
inline MsShape ms_shape(uint64_t n, uint64_t n_sources, int W, uint64_t resident) {
  const uint64_t batches = (n_sources + 64 * W - 1) / (64 * W);
  uint64_t groups = std::min(batches, resident * kMsNodesPerBlock / n);
  groups = std::min({groups, kMsMaskBytes / (n * W * 32), kMsGroups, resident});
  groups = std::max<uint64_t>(1, groups);
  const uint64_t rounds = (batches + groups - 1) / groups;  // as many groups as the rounds need
  groups = (batches + rounds - 1) / rounds;
  // fewer blocks make cheaper barriers
  const uint64_t want = (n + kMsBlockNodes - 1) / kMsBlockNodes;
  return MsShape{(uint32_t)groups, (uint32_t)std::max<uint64_t>(1, std::min(want, resident / groups))};
}

}  // namespace ug
