// Nodes that a build hands from one kernel to the next.  Plain host and
// device types, so that the width of their fields is checked on the host.
#pragma once

#include <stdint.h>

namespace pptkg {

// A segment for k_subtree.  Its parent is a record of any number below 2^31
// (a tree over 2^30 points has that many) or, for a cloud's root, -1 - cloud;
// the side is kept apart from it.
template <typename T, int D>
struct Small {
  int32_t b, e;
  int32_t parent;
  int16_t lvl, side;
  long long n_orig;  // input rows of the segment's cloud (the reference's num_points)
  T lo[D], hi[D];    // loose extent (the reference's node_box)
};

// A node of a subtree in shared memory: positions within its segment.
template <typename T, int D>
struct Entry {
  uint16_t b, e : 15, side : 1;
  int32_t parent;  // as Small's
  T lo[D], hi[D];
};

}  // namespace pptkg
