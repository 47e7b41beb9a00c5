// The 2D instances of the one-launch step.
#include "small.cuh"

namespace tsph {
template cudaError_t launch_small_dim<2>(tsph_ctx &, const SmallArgs &, int, cudaStream_t);
}  // namespace tsph
