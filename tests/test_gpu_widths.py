"""Kernels unrolled for widths 4 to 7 (eps 1e-3 .. 1e-6), 2D and 3D: forward
transform and trajectory gradients against the FP64 NDFT.

The gradient is Re(conj(dy) (-i) A(n_d x)) summed over coils.  The relative error
of a width-w kernel is about eps; bound 20 eps (the derivative of the kernel loses
about an order), the runtime-width kernels (w = 8, eps 1e-7; and 3D gradients) by
the same rule with FP32 rounding, 2e-5.
"""

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import ndft

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("shape,M", [((34, 48), 1001), ((20, 18, 16), 1501)])
@pytest.mark.parametrize("C", [1, 3])
def test_op_and_trajectory_gradient(gpu_pkg, eps, shape, M, C):
    rng = np.random.default_rng(M + C)
    d = len(shape)
    k = rng.uniform(-0.5, 0.5, (M, d)).astype(np.float32)
    k[:2] = -0.5
    cpx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    x, dy = cpx(1, C, *shape), cpx(1, C, M)
    op = gpu_pkg.MRIGB300(k, shape, n_coils=C, squeeze_dims=False, eps=eps)
    bound = max(20 * eps, 2e-5)
    ku, nrm = k.astype(np.float64), ndft.norm_factor(shape)
    ref = np.stack([ndft.ndft_type2(ku, x[0, c], shape) for c in range(C)]) / nrm
    assert rel_l2(op.op(x)[0], ref) < bound
    ag = op.make_autograd(wrt_data=True, wrt_traj=True)
    y = ag.op(torch.from_numpy(x).cuda())
    y.backward(torch.from_numpy(dy).cuda())
    g = np.zeros((M, d))
    for j in range(d):
        n = (np.arange(shape[j]) - shape[j] // 2).reshape([-1 if q == j else 1 for q in range(d)])
        for c in range(C):
            g[:, j] += (np.conj(dy[0, c]) * -1j * ndft.ndft_type2(ku, x[0, c] * n, shape)).real / nrm
    assert rel_l2(ag.samples.grad.cpu().numpy(), g) < bound
