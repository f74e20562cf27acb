// How many CTAs of a cluster share a sample (host only, no CUDA calls).
#pragma once
#include <cstdint>

namespace qsx {

// fits(c): whether c CTAs hold a sample; worth(c): whether 2 c of them would
// have work; clusters(c): how many clusters of c CTAs run at once, 0 also where
// the device does not answer.  As few CTAs as hold a sample, then twice as many
// while all samples still run at once; 0 when none can be scheduled.  A size
// that cannot be had is passed over: it is no error of the call.
template <class Fits, class Worth, class Clusters>
int choose_cluster(int64_t batch, int most, Fits fits, Worth worth, Clusters clusters) {
  int c = 1;
  while (c < most && !fits(c)) c *= 2;
  if (!fits(c) || clusters(c) < 1) return 0;
  while (c < most && worth(c) && clusters(2 * c) >= batch) c *= 2;
  return c;
}

}  // namespace qsx
