// Segment fluid kernels in double: the launch entry points of sweeps.cuh for this precision.
#include "seg_impl.cuh"

namespace img {
template cudaError_t launch_fluid_seg<double>(const FluidArgs&, const PencilLaunch&, int);
template cudaError_t launch_fluid_seg_batch<double>(const FluidArgs*, const BlockMap*, const PencilLaunch&, int);
template cudaError_t fluid_seg_attributes<double>(int);
}  // namespace img
