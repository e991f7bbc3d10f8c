// Groups the gates of a program into passes over the statevector.
//
// A gate pass reads and writes the whole statevector once, so a program of G
// dense gates of k <= 4 moves G times the state although each gate needs only
// 2^k amplitudes at a time.  A tile of 2^tb amplitudes held in shared memory can
// take every gate whose targets lie among the tile's tb qubits, one after the
// other, for one read and one write of the state.
//
// The grouping is greedy.  Every ready gate (no earlier pending gate shares a
// qubit with it) is tried as the seed of a tile; the tile grows by the ready
// gate that brings the most newly absorbed gates per added qubit until none
// fits; the seed whose tile absorbs the most gates becomes the next pass.  The
// scan looks at the first kWindow pending gates, which bounds the planning time
// of long programs (88 gates on 30 qubits: under 1 ms).
#include "pass_plan.hpp"

#include <algorithm>

namespace cb2 {

namespace {

constexpr size_t kWindow = 128;  // pending gates a scan looks at

uint32_t count_bits(uint64_t x) { return (uint32_t)__builtin_popcountll(x); }

struct Scan {
  uint32_t taken = 0;
  uint64_t ready[64];  // target masks of ready mergeable gates outside the tile
  uint32_t n_ready = 0;
};

// Walks the pending gates for tile `q`: a gate is taken when it fits and nothing
// before it that stays behind shares a qubit.  `out` (may be null) receives the
// indices taken.
void scan(const std::vector<PassGate> &g, const std::vector<uint32_t> &pending, uint64_t q,
          uint64_t all, uint32_t max_gates, Scan &s, std::vector<uint32_t> *out) {
  s.taken = s.n_ready = 0;
  uint64_t blocked = 0;
  const size_t end = std::min(pending.size(), kWindow);
  for (size_t i = 0; i < end && (all & ~blocked); ++i) {
    const PassGate &x = g[pending[i]];
    if (!(x.qubits & blocked) && x.mergeable) {
      if (!(x.qubits & ~q) && s.taken < max_gates) {
        ++s.taken;
        if (out) out->push_back(pending[i]);
        continue;
      }
      if ((x.qubits & ~q) && s.n_ready < 64) s.ready[s.n_ready++] = x.qubits;
    }
    blocked |= x.qubits;
  }
}

}  // namespace

std::vector<Pass> plan_passes(const std::vector<PassGate> &g, uint32_t n, uint32_t tb, uint32_t low,
                              uint32_t max_gates, uint32_t cost) {
  std::vector<Pass> out;
  std::vector<uint32_t> pending(g.size());
  for (uint32_t i = 0; i < g.size(); ++i) pending[i] = i;
  const uint64_t all = n >= 64 ? ~0ull : (1ull << n) - 1;
  const uint64_t low_mask = (1ull << std::min(low, n)) - 1;
  Scan s, t;
  while (!pending.empty()) {
    Pass best;
    scan(g, pending, low_mask, all, max_gates, s, nullptr);
    std::vector<uint64_t> seeds(s.ready, s.ready + s.n_ready);
    if (s.taken) seeds.push_back(low_mask);
    uint32_t best_taken = 0;
    for (const uint64_t seed : seeds) {
      uint64_t q = low_mask | seed;
      if (count_bits(q) > tb) continue;
      scan(g, pending, q, all, max_gates, s, nullptr);
      while (s.n_ready) {
        uint64_t grow = 0;
        uint32_t gain = 0, added = 1;
        for (uint32_t c = 0; c < s.n_ready; ++c) {
          const uint64_t qq = q | s.ready[c];
          if (count_bits(qq) > tb) continue;
          scan(g, pending, qq, all, max_gates, t, nullptr);
          const uint32_t more = t.taken - std::min(t.taken, s.taken), add = count_bits(qq) - count_bits(q);
          if (more && (!grow || more * added > gain * add)) {
            grow = qq;
            gain = more;
            added = add;
          }
        }
        if (!grow) break;
        q = grow;
        scan(g, pending, q, all, max_gates, s, nullptr);
      }
      if (s.taken > best_taken) {
        best_taken = s.taken;
        best.tile = q;
      }
    }
    uint32_t saved = 0;
    if (best_taken >= 2) {
      scan(g, pending, best.tile, all, max_gates, s, &best.gates);
      for (const uint32_t i : best.gates) saved += g[i].saves;
    }
    if (saved < cost) {
      best.tile = 0;  // nothing to merge now: the oldest pending gate runs alone
      best.gates.assign(1, pending[0]);
    }
    std::vector<uint32_t> rest;
    rest.reserve(pending.size());
    size_t j = 0;
    for (const uint32_t i : pending) {
      if (j < best.gates.size() && best.gates[j] == i) ++j;
      else rest.push_back(i);
    }
    pending.swap(rest);
    if (best.tile)  // spare tile qubits: the lowest free ones (longer contiguous runs)
      for (uint32_t b = 0; b < n && count_bits(best.tile) < tb; ++b) best.tile |= 1ull << b;
    out.push_back(std::move(best));
  }
  return out;
}

}  // namespace cb2
