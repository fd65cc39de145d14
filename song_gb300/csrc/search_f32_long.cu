// search_f32_long.cu -- the FP32 search: rows of LONG_ROW bytes and more.
#include "search_kernel.cuh"

namespace song {
int launch_f32_long(const Params &p, int metric, int S, cudaStream_t s) {
  return launch_storage<0, false, false, true>(p, metric, S, s);
}
}  // namespace song
