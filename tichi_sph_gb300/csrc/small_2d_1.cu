// The one-launch step in 2D with 1 lane per particle.
#include "small.cuh"

namespace tsph {
template cudaError_t launch_small_lanes<2, 1, false>(tsph_ctx &, const SmallArgs &, int, cudaStream_t);
}  // namespace tsph
