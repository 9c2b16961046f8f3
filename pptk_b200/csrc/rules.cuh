// Choices of the kNN and normal walks by sizes and settings.  Plain functions,
// compiled for the host by a test.
#pragma once

#include <stdint.h>

namespace pptkg {

// Window of a packet's warm lists, in multiples of k: one more than the
// warm_mult setting where packets span over 256 tree positions and lists are
// short.  Their queries' walks share less, so candidates found before them
// save more (1M scattered queries, k = 16: 2.35 -> 2.10 ms; queries in tree
// order: 31.8 -> 32.7).  A setting of 1 is the k-position start everywhere.
inline int warm_window(int mult, int64_t nv, int64_t m, int kmax) {
  return mult + (mult > 1 && kmax <= 16 && 32 * nv > 256 * m ? 1 : 0);
}

}  // namespace pptkg
