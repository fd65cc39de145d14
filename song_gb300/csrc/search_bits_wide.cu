// search_bits_wide.cu -- the search over codes of vectors whose FP32 query is
// staged for the re-rank only (WarpLayout).
#include "search_kernel.cuh"

namespace song {
int launch_bits_wide(const Params &p, int metric, int S, cudaStream_t s) {
  return launch_storage<3, false, false, true>(p, metric, S, s);
}
}  // namespace song
