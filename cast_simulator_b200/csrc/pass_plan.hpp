// Grouping of a gate program's gates into passes over the statevector (host only).
#pragma once

#include <cstdint>
#include <vector>

namespace cb2 {

constexpr uint32_t kMaxPassGates = 16;  // gates one merged pass applies

struct PassGate {
  uint64_t qubits = 0;     // target mask
  bool mergeable = false;  // may share a pass with others (else it runs alone)
  uint32_t saves = 10;     // what sharing a pass saves, in tenths of a one-gate pass
};

// One pass: a single gate on its own kernel (tile == 0), or several gates applied
// to tiles of 2^tb amplitudes whose qubits are `tile` (a superset of every
// gate's targets, holding the `low` lowest qubits).
struct Pass {
  std::vector<uint32_t> gates;  // indices into the program, in execution order
  uint64_t tile = 0;
};

// Partitions `gates` (program order) into passes for tiles of tb qubits.  Gates
// that share a qubit keep their order; gates on disjoint qubits commute.
// At most max_gates (<= kMaxPassGates) share a pass, and only if together they
// save at least `cost` (tenths of a one-gate pass).
std::vector<Pass> plan_passes(const std::vector<PassGate> &gates, uint32_t n, uint32_t tb,
                              uint32_t low, uint32_t max_gates, uint32_t cost);

}  // namespace cb2
