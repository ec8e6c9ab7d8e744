// Whether a cluster kernel can run on the device at hand, from the runtime's
// answers (host code; the calls come in as functions).
#pragma once

namespace ilbm {

// prepare: sets the kernel's attributes (opt-in shared memory, cluster size);
// query: clusters of it that can be resident at once; clear: drops the error a
// refusal leaves behind.  prepare and query return 0 on success.  A device or
// partition that refuses the attributes, or holds no such cluster, is no error:
// the caller takes its launches without clusters.
template <class Prepare, class Query, class Clear>
inline bool cluster_fits(Prepare prepare, Query query, Clear clear) {
  int resident = 0;
  if (prepare() == 0 && query(&resident) == 0) return resident > 0;
  clear();
  return false;
}

}  // namespace ilbm
