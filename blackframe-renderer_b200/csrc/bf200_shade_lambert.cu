// The Lambert route's shading kernels, with their building blocks inlined.
#define BF_SHADE_INLINE
#include "bf200_kernels_body.cuh"

namespace bf200 {
#define BF200_SHADE_LAMBERT(ADJ, CONE, TREE)                                                                      \
    template void launch_shade_lambert<ADJ, CONE, TREE>(const SceneView&, const Wavefront&, const PathSource&,   \
                                                        const TransportParams&, uint32_t, const AdjointView&,    \
                                                        cudaStream_t);
BF200_SHADE_LAMBERT(false, false, false)
BF200_SHADE_LAMBERT(false, true, false)
BF200_SHADE_LAMBERT(false, false, true)
BF200_SHADE_LAMBERT(false, true, true)
BF200_SHADE_LAMBERT(true, false, false)
#undef BF200_SHADE_LAMBERT
}  // namespace bf200
