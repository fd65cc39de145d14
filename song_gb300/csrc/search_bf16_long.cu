// search_bf16_long.cu -- the BF16 search: rows of LONG_ROW bytes and more.
#include "search_kernel.cuh"

namespace song {
int launch_bf16_long(const Params &p, int metric, int S, cudaStream_t s) {
  return launch_storage<1, false, false, true>(p, metric, S, s);
}
}  // namespace song
