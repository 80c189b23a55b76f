// Trajectory-gradient kernels (2D and 3D).
#include "gbn_kernels.cuh"

namespace gbn {
cudaError_t launch_grad2d(const GradArgs& a, cudaStream_t st) { return dispatch_grad<2>(a, st); }
cudaError_t launch_grad3d(const GradArgs& a, cudaStream_t st) { return dispatch_grad<3>(a, st); }
}  // namespace gbn
