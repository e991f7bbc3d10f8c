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
// of long programs: a pass costs what its window does, however many gates wait
// behind it.  Tiles that another seed has already grown through are not grown
// again, and a count ends where the tile's qubits are all blocked.  2000 1-qubit
// gates on 20 qubits 0.5 ms (30 without these), 50000 14 ms (0.9 s), 600 on 30 qubits
// 0.6 ms (24), unfused brickwork of depth 20 on 28 qubits 0.4 ms (7).
#include "pass_plan.hpp"

#include <algorithm>

namespace cb2 {

namespace {

constexpr size_t kWindow = 128;  // pending gates a scan looks at

uint32_t count_bits(uint64_t x) { return (uint32_t)__builtin_popcountll(x); }

// The first pending gates, and how many a pass may take.
struct Window {
  uint64_t qubits[kWindow];
  bool mergeable[kWindow];
  uint32_t n = 0, max_gates = 0;
  uint64_t all = 0;  // every qubit
};

struct Scan {
  uint32_t taken = 0;
  uint64_t ready[64];  // target masks of ready mergeable gates outside the tile
  uint32_t n_ready = 0;
};

// Walks the window for tile `q`: a gate is taken when it fits and nothing before it
// that stays behind shares a qubit.  `out` (may be null) receives the places taken.
void scan(const Window &w, uint64_t q, Scan &s, std::vector<uint32_t> *out) {
  s.taken = s.n_ready = 0;
  uint64_t blocked = 0;
  for (uint32_t i = 0; i < w.n && (w.all & ~blocked); ++i) {
    const uint64_t x = w.qubits[i];
    if (!(x & blocked) && w.mergeable[i]) {
      if (!(x & ~q) && s.taken < w.max_gates) {
        ++s.taken;
        if (out) out->push_back(i);
        continue;
      }
      if ((x & ~q) && s.n_ready < 64) s.ready[s.n_ready++] = x;
    }
    blocked |= x;
  }
}

// How many gates scan takes.
uint32_t count(const Window &w, uint64_t q) {
  uint32_t taken = 0;
  uint64_t blocked = 0;
  for (uint32_t i = 0; i < w.n && (q & ~blocked) && taken < w.max_gates; ++i) {
    const uint64_t x = w.qubits[i];
    if (!(x & (blocked | ~q)) && w.mergeable[i]) ++taken;
    else blocked |= x;
  }
  return taken;
}

}  // namespace

std::vector<Pass> plan_passes(const std::vector<PassGate> &g, uint32_t n, uint32_t tb, uint32_t low,
                              uint32_t max_gates, uint32_t cost) {
  std::vector<Pass> out;
  // pending gates: those left of the window (program order), then `next` and on
  uint32_t pending[kWindow];
  uint32_t next = 0;
  Window w;
  w.all = n >= 64 ? ~0ull : (1ull << n) - 1;
  w.max_gates = max_gates;
  const uint64_t low_mask = (1ull << std::min(low, n)) - 1;
  Scan s;
  std::vector<uint64_t> seeds, seen;
  std::vector<uint32_t> places;
  for (;;) {
    for (; w.n < kWindow && next < g.size(); ++next, ++w.n) {
      pending[w.n] = next;
      w.qubits[w.n] = g[next].qubits;
      w.mergeable[w.n] = g[next].mergeable;
    }
    if (!w.n) break;
    Pass best;
    scan(w, low_mask, s, nullptr);
    seeds.assign(s.ready, s.ready + s.n_ready);
    if (s.taken) seeds.push_back(low_mask);
    seen.clear();
    uint32_t best_taken = 0;
    for (size_t j = 0; j < seeds.size() && best_taken < max_gates; ++j) {
      uint64_t q = low_mask | seeds[j];
      if (count_bits(q) > tb) continue;
      // a tile grown through before would end as it did then
      auto grown = [&] { return std::find(seen.begin(), seen.end(), q) != seen.end(); };
      if (grown()) continue;
      seen.push_back(q);
      scan(w, q, s, nullptr);
      bool known = false;
      while (s.n_ready && s.taken < max_gates) {
        uint64_t grow = 0;
        uint32_t gain = 0, added = 1;
        for (uint32_t c = 0; c < s.n_ready; ++c) {
          const uint64_t qq = q | s.ready[c];
          if (count_bits(qq) > tb) continue;
          const uint32_t t = count(w, qq), more = t - std::min(t, s.taken), add = count_bits(qq) - count_bits(q);
          if (more && (!grow || more * added > gain * add)) {
            grow = qq;
            gain = more;
            added = add;
          }
        }
        if (!grow) break;
        q = grow;
        if ((known = grown())) break;
        seen.push_back(q);
        scan(w, q, s, nullptr);
      }
      if (!known && s.taken > best_taken) {
        best_taken = s.taken;
        best.tile = q;
      }
    }
    uint32_t saved = 0;
    places.clear();
    if (best_taken >= 2) {
      scan(w, best.tile, s, &places);
      for (const uint32_t i : places) saved += g[pending[i]].saves;
    }
    if (saved < cost) {
      best.tile = 0;  // nothing to merge now: the oldest pending gate runs alone
      places.assign(1, 0);
    }
    uint32_t kept = 0;
    size_t j = 0;
    for (uint32_t i = 0; i < w.n; ++i) {
      if (j < places.size() && places[j] == i) {
        best.gates.push_back(pending[i]);
        ++j;
        continue;
      }
      pending[kept] = pending[i];
      w.qubits[kept] = w.qubits[i];
      w.mergeable[kept++] = w.mergeable[i];
    }
    w.n = kept;
    if (best.tile)  // spare tile qubits: the lowest free ones (longer contiguous runs)
      for (uint32_t b = 0; b < n && count_bits(best.tile) < tb; ++b) best.tile |= 1ull << b;
    out.push_back(std::move(best));
  }
  return out;
}

}  // namespace cb2
