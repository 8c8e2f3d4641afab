// Window magnet kernels in float: the launch entry points of sweeps.cuh for this precision.
#include "seg_impl.cuh"

namespace img {
template cudaError_t launch_mag_chain_win<float>(const MagArgs&, const PencilLaunch&);
template cudaError_t launch_mag_ct_win<float>(const MagArgs&, const PencilLaunch&);
template cudaError_t launch_mag_chain_win_batch<float>(const MagArgs*, const BlockMap*, const PencilLaunch&);
template cudaError_t launch_mag_ct_win_batch<float>(const MagArgs*, const BlockMap*, const PencilLaunch&);
template cudaError_t chain_win_attributes<float>(int);
}  // namespace img
