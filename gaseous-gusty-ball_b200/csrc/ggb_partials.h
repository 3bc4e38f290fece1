// ggb_partials.h — where the solve kernel's blocks leave their sums at a grid
// barrier (vsync in solver_body.cuh).  Plain C++, so that the rule can be checked
// on the host.
#pragma once

#include <cstddef>

namespace ggb {

// The barriers of a solve take the sets of partials in turn.  A block writes its
// row of barrier e's set before it arrives at e.  The rows are read after e and
// before the reader arrives at e + 1; a late sum is read beside barrier e + 1, with
// nothing between that read and the reader's own arrival at e + 1, and so is only
// known to be over when the reader arrives at e + 2.  A block writes for barrier w
// when it has passed w - 1, where all blocks have arrived.  The next write to a set
// therefore has to be at e + 2 or later for a sum read at once and at e + 3 or later
// for a late one: three sets.  (With two, a block that had passed e + 1 could put
// its sum of psi in the place of its |r|^2 under another block's late read.)
constexpr int kPartSets = 3;
constexpr int part_set(int epoch) { return epoch % kPartSets; }

// Doubles of the partials of a solve on at most `blocks` blocks: two sums a set.
constexpr size_t part_doubles(int blocks) { return (size_t)kPartSets * 2 * blocks; }

}  // namespace ggb
