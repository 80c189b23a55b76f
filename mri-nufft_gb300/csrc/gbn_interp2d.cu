// 2D instantiations of the interpolation kernels.
#include "gbn_kernels.cuh"

namespace gbn {
cudaError_t launch_interp2d(const InterpArgs& a, cudaStream_t st) { return dispatch_interp<2>(a, st); }
}  // namespace gbn
