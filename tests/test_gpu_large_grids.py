"""Grids whose sort has more than 4096 x 4096 keys, where the scan of the bin
counts takes a third level: 1024^3 cells (a 512^3 image, the Toeplitz kernel of a
256^3 one), plans of two transforms from 13 000^2 cells on, bins of one cell.

Bounds: the same kernels in another order of samples agree to FP32 rounding of
sums, 1e-5 relative l2; adjointness to 1e-5 of the product.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _samples(M, dim, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = (torch.rand(M, dim, generator=g, device="cuda") - 0.5) * (2 * np.pi)
    k[:4] = -np.pi
    k[4:8] = float(np.nextafter(np.float32(np.pi), np.float32(0)))
    return k


def _cpx(*s):
    return torch.randn(*s, dtype=torch.complex64, device="cuda")


def test_cells_of_a_512_cubed_image(gpu_pkg):
    k = _samples(4096, 3, 0)
    plan = gpu_pkg.NufftPlan((1024, 1024, 1024), spread_only=True)
    plan.setpts(k)
    y = _cpx(1, k.shape[0])
    grid = torch.empty((1024, 1024, 1024), dtype=torch.complex64, device="cuda")
    plan.adj(y, None, None, grid, 1, 1, 1.0)
    back = torch.empty_like(y)
    plan.op(grid, None, back, 1, 1, 1.0)
    norm2 = torch.view_as_real(grid).square().sum(dtype=torch.float64).item()
    dot = torch.vdot(y[0].to(torch.complex128), back[0].to(torch.complex128))
    assert abs(dot.real.item() - norm2) < 1e-5 * norm2
    assert abs(dot.imag.item()) < 1e-5 * norm2


@pytest.mark.parametrize("shape,ntrans,bins", [((2080, 2080), 1, (1, 1)), ((6500, 6520), 2, None)])
def test_more_keys_than_two_scan_levels(gpu_pkg, monkeypatch, shape, ntrans, bins):
    k = _samples(3000, 2, 1)
    plan = gpu_pkg.NufftPlan(shape, ntrans=ntrans)
    if bins:
        plan.tune(bins=bins)
    info = plan.info()
    assert -(-info["nf"][0] // info["bins"][0]) * info["nf"][1] > 4096 * 4096
    plan.setpts(k)
    monkeypatch.setenv("GBN_SPREAD", "gm")  # its bins are wider: fewer keys
    ref = gpu_pkg.NufftPlan(shape, ntrans=ntrans)
    ref.setpts(k)
    x, y = _cpx(ntrans, *shape), _cpx(ntrans, k.shape[0])
    out = []
    for p in (plan, ref):
        out.append((p.op(x, None, torch.empty_like(y), 1, ntrans, 1.0),
                    p.adj(y, None, None, torch.empty_like(x), 1, ntrans, 1.0)))
    for a, b in zip(*out):
        assert (torch.linalg.norm(a - b) / torch.linalg.norm(b)).item() < 1e-5
