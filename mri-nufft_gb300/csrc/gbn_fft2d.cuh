// Pruned 2D transforms fused with the pad / crop passes (see gbn_fft2d.cu).
#pragma once

#include "gbn_fft3d.cuh"
#include "gbn_passes.cuh"

namespace gbn {

// 2D plans whose fine grid has 256, 384, 512, 640 or 768 cells on both axes
bool fft2d_fits(const Geom& g);

// raises the dynamic shared-memory limit of the plan's kernels (once, outside any
// stream capture)
cudaError_t fft2d_prepare(const Geom& g);

// op: pad and the pruned transform of sign isign into pa.fine (pa.ntr
// grids); every fine cell is written.
cudaError_t launch_fft2d_op(const PadArgs& pa, const Twiddles& tw, int isign, cudaStream_t st);

// adjoint: the pruned transform of sign isign of `fine` (ca.ntr grids, read
// and overwritten) and the crop / coil combine of ca into ca.out.
cudaError_t launch_fft2d_adj(const CropArgs& ca, float2* fine, const Twiddles& tw, int isign,
                             cudaStream_t st);

// Toeplitz Gram of a pass: pad, forward transform, multiply by the real
// circulant spectrum K (512-point x axis), inverse transform and crop, with the
// x transforms and the multiply in one pass over the y columns.
cudaError_t launch_fft2d_gram(const PadArgs& pa, const CropArgs& ca, const float* K,
                              const Twiddles& tw, cudaStream_t st);

}  // namespace gbn
