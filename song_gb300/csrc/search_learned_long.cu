// search_learned_long.cu -- the learned search: rows of LONG_ROW bytes and more.
#include "search_kernel.cuh"

namespace song {
int launch_learned_long(const Params &p, int storage, int metric, int S, cudaStream_t s) {
  if (storage == 0) return launch_storage<0, true, false, true>(p, metric, S, s);
  if (storage == 1) return launch_storage<1, true, false, true>(p, metric, S, s);
  return -1;
}
}  // namespace song
