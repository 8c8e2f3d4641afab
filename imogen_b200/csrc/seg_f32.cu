// Segment fluid kernels in float: the launch entry points of sweeps.cuh for this precision.
#include "seg_impl.cuh"

namespace img {
template cudaError_t launch_fluid_seg<float>(const FluidArgs&, const PencilLaunch&, int);
template cudaError_t launch_fluid_seg_batch<float>(const FluidArgs*, const BlockMap*, const PencilLaunch&, int);
template cudaError_t fluid_seg_attributes<float>(int);
}  // namespace img
