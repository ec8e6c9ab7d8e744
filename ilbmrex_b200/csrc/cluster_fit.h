// How many clusters of a kernel the device at hand runs at once, from the
// runtime's answers (host code; the calls come in as functions).
#pragma once

namespace ilbm {

// prepare: sets the kernel's attributes (opt-in shared memory, cluster size);
// query: clusters of it that can be resident at once; clear: drops the error a
// refusal leaves behind.  prepare and query return 0 on success.  A device or
// partition that refuses the attributes, or holds no such cluster, is no error
// but 0: the caller takes its launches without clusters.
template <class Prepare, class Query, class Clear>
inline int clusters_resident(Prepare prepare, Query query, Clear clear) {
  int resident = 0;
  if (prepare() == 0 && query(&resident) == 0) return resident > 0 ? resident : 0;
  clear();
  return 0;
}

}  // namespace ilbm
