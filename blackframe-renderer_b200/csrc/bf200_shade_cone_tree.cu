// Shading kernels of cone-carrying traces of tree-selecting scenes.
#include "bf200_kernels_body.cuh"

namespace bf200 {
template void launch_shade_others<false, true, true>(const SceneView&, const Wavefront&, const PathSource&, const TransportParams&,
                                    uint32_t, const AdjointView&, const cudaStream_t (&)[kShadeBranches]);
}  // namespace bf200
