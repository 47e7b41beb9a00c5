// The one-launch step in 3D with one lane per particle, warps with several runs each.
#include "small.cuh"

namespace tsph {
template cudaError_t launch_small_lanes<3, 1, true>(tsph_ctx &, const SmallArgs &, int, cudaStream_t);
}  // namespace tsph
