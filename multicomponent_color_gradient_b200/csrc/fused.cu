// fused.cu - the fused step's kernels of one row pitch MCG_PITCH (0: runtime).
#include "fused.cuh"

namespace mcg {
template cudaError_t fused_configure_pitch<MCG_PITCH>(const Geometry &, const FusedTiling &);
template cudaError_t fused_launch_pitch<MCG_PITCH>(const DeviceState &, const FusedTiling &, int, int64_t, bool,
                                                   cudaStream_t);
template cudaError_t moments_launch_pitch<MCG_PITCH>(const DeviceState &, int, int64_t, int, int, cudaStream_t);
template cudaError_t collide_launch_pitch<MCG_PITCH>(const DeviceState &, int, int64_t, cudaStream_t);
}  // namespace mcg
