// Which blocks of a trajectory program share passes (host only).
#pragma once

#include <cstdint>
#include <vector>

#include "pass_plan.hpp"

namespace cb2 {

// A fused block and the Pauli error sites behind it.
struct SegBlock {
  uint64_t qubits = 0;
  double quiet = 1;        // chance that none of its sites fires
  bool follows = false;    // directly behind the block before it (no damping or channel between)
};

// Blocks first .. first + count - 1 as passes, taken when none of their sites fires.
struct Segment {
  uint32_t first = 0, count = 0;
  std::vector<Pass> passes;  // gates: indices from `first`
};

// The segments that pay, in order; none where the program as a whole is better off
// in the plain kernel.
std::vector<Segment> plan_segments(const std::vector<SegBlock> &blocks, uint32_t n, uint32_t tb, uint32_t low);

// Mean qubits of the blocks (0 without blocks).
double mean_width(const std::vector<SegBlock> &blocks);

// Threads a CTA for blocks in place (see seg_plan.cpp).
unsigned plain_threads(uint32_t n, double width);

}  // namespace cb2
