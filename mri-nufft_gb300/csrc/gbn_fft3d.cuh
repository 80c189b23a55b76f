// Pruned 3D transforms fused with the pad / crop passes (see gbn_fft3d.cu).
#pragma once

#include <vector>

#include "gbn_passes.cuh"

namespace gbn {

// 3D plans whose fine grid has 128, 192 or 256 cells on every axis
bool fft3d_fits(const Geom& g);

// W_n^(b k1), entry k1 * 16 + b (k1 < n / 16, b < 16), as 2 n floats (re, im)
std::vector<float> fft_twiddles(int n);

// device tables of fft_twiddles, one per axis
struct Twiddles {
  const float2* t[3];
};

// raises the dynamic shared-memory limit of the crop kernels (once, outside
// any stream capture)
cudaError_t fft3d_prepare();

// op: pad (pa: image, coil maps, 1/phihat, scale) and the pruned transform
// of sign isign into pa.fine (pa.ntr grids); every fine cell is written.
cudaError_t launch_fft3d_op(const PadArgs& pa, const Twiddles& tw, int isign, cudaStream_t st);

// adjoint: the pruned transform of sign isign of `fine` (ca.ntr grids, read
// and overwritten) and the crop / coil combine of ca into ca.out.
cudaError_t launch_fft3d_adj(const CropArgs& ca, float2* fine, const Twiddles& tw, int isign,
                              cudaStream_t st);

// Toeplitz Gram of a pass (pa.ntr = ca.ntr transforms): pad, forward
// transform, multiply by the real circulant spectrum K (256-point x axis), inverse
// transform and crop, with the x transforms and the multiply in one pass
// over the (y, z) lines; the fine grids hold only intermediate line data.
cudaError_t launch_fft3d_gram(const PadArgs& pa, const CropArgs& ca, const float* K,
                               const Twiddles& tw, cudaStream_t st);

}  // namespace gbn
