"""Fused line transforms of every axis length, mixed and with odd image sizes.

3D fine grids of 128, 192 or 256 cells an axis and 2D ones of 256, 384, 512, 640
or 768 run fused pad / transform / crop passes; GBN_FUSED_FFT=0 keeps cuFFT.  Both
compute the same sums in FP32: relative l2 <= 1e-5 (the bound of the 256^3 and
512^2 tests) for op, adjoint, data consistency, the Gram operator and the +1 sign.
"""

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu

SAME = 1e-5


@pytest.mark.parametrize("shape", [(64, 64, 64), (96, 96, 96), (64, 96, 128), (128, 63, 95), (127, 128, 64),
                                   (128, 128), (192, 192), (320, 320), (384, 384), (128, 383), (319, 192),
                                   (256, 127), (253, 320)])
@pytest.mark.parametrize("sense,C", [(True, 5), (False, 1)])
def test_fused_equals_cufft_path(gpu_pkg, monkeypatch, shape, sense, C):
    rng = np.random.default_rng(sum(shape) + C)
    M = 5000
    k = rng.uniform(-0.5, 0.5, (M, len(shape))).astype(np.float32)
    cpx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    smaps = cpx(C, *shape) if sense else None
    x, y = cpx(1, 1 if sense else C, *shape), cpx(1, C, M)
    dens = rng.uniform(0.5, 1.5, M).astype(np.float32)
    res = []
    for env in ("1", "0"):
        monkeypatch.setenv("GBN_FUSED_FFT", env)
        op = gpu_pkg.MRIGB300(k, shape, n_coils=C, smaps=smaps, density=dens, squeeze_dims=False)
        r = [op.op(x), op.adj_op(y), op.data_consistency(x, y), op.gram_op(x)]
        xt = torch.from_numpy(x).cuda()
        out = torch.empty((1, C, M), dtype=torch.complex64, device="cuda")
        op.plan.op(xt, op._smaps, out, 1, C, 1.0, isign=+1)
        img = torch.empty(xt.shape, dtype=torch.complex64, device="cuda")
        op.plan.adj(torch.from_numpy(y).cuda(), None, op._smaps, img, 1, C, 1.0, isign=-1)
        res.append(r + [out.cpu().numpy(), img.cpu().numpy()])
    for a, b in zip(*res):
        assert rel_l2(a, b) < SAME
