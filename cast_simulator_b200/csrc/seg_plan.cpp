// Segments of a trajectory program: pieces of it whose blocks share passes over the
// state whenever no error site of the piece fires.
//
// How long a piece should be and whether it pays depends on how often it fires: a
// fired piece runs block by block, in a kernel that is no better at that than the
// plain one.  2072 trajectories of 13 qubits, depth 30, fused at 2, error rate 1e-2
// without damping: plain kernel 10.9 ms, the circuit as one segment 13.0, in pieces
// 8.7; at 1e-1, where none pays, 16.5 and 19.0.
#include "seg_plan.hpp"

#include <cmath>

namespace cb2 {

namespace {

// What a piece of a program costs, in blocks run in place by the plain kernel.  A
// segment draws for its sites (`draw`), then makes its passes (start and copies
// `pass`, a block in the tile kTile).  Where a site fires its blocks run in place,
// which in this kernel costs `in_place`: from 13 qubits the tiles' shared memory takes
// the L1 that held the state, at 17 narrow blocks miss the loads in flight of 1024
// threads.  Fitted to brickwork of 8 to 18 qubits fused at 2, 3 and 4 with error
// rates of 1e-3 to 1e-1, with and without damping layers.
struct SegCost {
  static constexpr double kTile = 0.42;
  double draw, pass, in_place;
  SegCost(uint32_t n, double width) {
    // a narrow block: 3 us at 12 qubits, 60 at 17
    draw = n <= 12 ? 0.3 : n <= 14 ? 0.5 : 0.25;
    pass = n <= 14 ? 1.4 : n == 15 ? 1.2 : 0.7;
    in_place = n <= 12 ? 1.08 : n <= 14 ? 1.15 : plain_threads(n, width) == 1024 && n == 17 ? 1.25 : 1.0;
    pass /= std::exp2(0.5 * (width - 2));  // a block of 4 qubits takes twice one of 2
  }
  // `quiet`: how often no site of the piece fires
  double segment(double quiet, double blocks, double passes) const {
    return draw + quiet * (pass * passes + kTile * blocks) + (1 - quiet) * in_place * blocks;
  }
  // The best length of a piece: longer ones share their draws and pass among more
  // blocks, but fire more often.  A piece ends before -log(quiet) * blocks passes this.
  double cut() const { return (draw + pass) / (in_place - kTile); }
};

}  // namespace

double mean_width(const std::vector<SegBlock> &blocks) {
  double width = 0;
  for (const SegBlock &b : blocks) width += __builtin_popcountll(b.qubits);
  return blocks.empty() ? 0 : width / (double)blocks.size();
}

// 512, whose registers the gate arithmetic needs, except where states are held in L2
// and blocks are narrow: passes bound by loads in flight.  1024 against 512 threads,
// noisy brickwork: 17 qubits, width 1.9 41.1 and 51.4 ms, 3.4 39.0 and 39.6, 3.7 18.5
// and 16.7; 16 qubits, 2.0 41.2 and 43.6, 2.1 45.4 and 44.9, 3.6 56.4 and 45.4; 15
// qubits, 1.9 22.8 and 21.6.
unsigned plain_threads(uint32_t n, double width) {
  return (n == 16 && width <= 2) || (n == 17 && width <= 3.5) ? 1024u : 512u;
}

std::vector<Segment> plan_segments(const std::vector<SegBlock> &blocks, uint32_t n, uint32_t tb, uint32_t low) {
  std::vector<Segment> out;
  const SegCost cost(n, mean_width(blocks));
  double expected = cost.in_place * (double)blocks.size();  // of the whole program
  for (uint32_t i = 0; i < blocks.size();) {
    Segment s;
    s.first = i;
    double quiet = 1;
    std::vector<PassGate> gates;
    do {
      const double with = quiet * blocks[i].quiet;
      if (s.count && !(-std::log(with) * (s.count + 1) <= cost.cut())) break;
      quiet = with;
      PassGate g;
      g.qubits = blocks[i].qubits;
      g.mergeable = true;
      gates.push_back(g);
      ++s.count;
      ++i;
    } while (i < blocks.size() && blocks[i].follows);
    s.passes = plan_passes(gates, n, tb, low, kMaxPassGates, 11);
    const double merged = cost.segment(quiet, s.count, (double)s.passes.size());
    const double in_place = cost.in_place * s.count;
    if (s.passes.size() >= s.count || merged >= in_place) continue;
    expected += merged - in_place;
    out.push_back(std::move(s));
  }
  if (expected >= 0.98 * (double)blocks.size()) out.clear();
  return out;
}

}  // namespace cb2
