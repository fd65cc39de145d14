// search_multi_long.cu -- the multi-probe search: rows of LONG_ROW bytes and more.
#include "search_kernel.cuh"

namespace song {
int launch_multi_long(const Params &p, int metric, int S, cudaStream_t s) {
  return launch_storage<0, false, true, true>(p, metric, S, s);
}
}  // namespace song
