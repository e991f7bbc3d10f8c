// Prints the segments of a program of equal 2-qubit blocks in brickwork order:
// argv: qubits, layers, chance that a block stays quiet, 1 when layers end in damping.
#include "seg_plan.hpp"

#include <cstdio>
#include <cstdlib>

int main(int, char **argv) {
  const unsigned n = (unsigned)std::atoi(argv[1]), layers = (unsigned)std::atoi(argv[2]);
  std::vector<cb2::SegBlock> blocks;
  for (unsigned l = 0; l < layers; ++l)
    for (unsigned q = l & 1; q + 1 < n; q += 2) {
      cb2::SegBlock b;
      b.qubits = 3ull << q;
      b.quiet = std::atof(argv[3]);
      b.follows = !blocks.empty() && (q > (l & 1) || argv[4][0] == '0');
      blocks.push_back(b);
    }
  for (const cb2::Segment &s : cb2::plan_segments(blocks, n, n < 13 ? n : 13, 4))
    std::printf("%u %u %zu\n", s.first, s.count, s.passes.size());
  std::printf("%zu %u\n", blocks.size(), cb2::plain_threads(n, cb2::mean_width(blocks)));
  return 0;
}
