"""Spreading and interpolation on grids smaller than the kernel, where footprints wrap
around several times, and samples at both ends of the period, against the kernel summed
in double precision (spread-only plans).  Bound: FP32 kernel values, 2e-6 relative l2
(2e-7 a weight, up to three factors)."""

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _axis(k, n, w, beta):
    """(M, n) weights of samples k (radians) on a periodic axis of n cells."""
    u = (k.astype(np.float64) / (2 * np.pi)) % 1.0 * n
    out = np.zeros((len(k), n))
    first = np.ceil(u - w / 2).astype(int)
    for t in range(w):
        z = (first + t - u) / (w / 2)
        v = np.exp(beta * (np.sqrt(np.maximum(1 - z * z, 0)) - 1)) * (z * z < 1)
        np.add.at(out, (np.arange(len(k)), (first + t) % n), v)
    return out


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("shape", [(1, 1), (1, 2), (3, 4), (5, 9), (8, 16), (17, 33), (1, 1, 1), (2, 3, 1), (4, 8, 16),
                                   (9, 7, 10)])
def test_footprints_that_wrap(gpu_pkg, shape, eps):
    rng = np.random.default_rng(len(shape))
    M, d = 64, len(shape)
    # whole cells and halves are where the first cell changes: stay 1e-3 of a cell away
    u = np.floor(rng.uniform(0, 1, (M, d)) * np.array(shape) * 2) / 2 + rng.uniform(1e-3, 0.499, (M, d))
    k = ((u / np.array(shape) * 2 * np.pi + np.pi) % (2 * np.pi) - np.pi).astype(np.float32)
    plan = gpu_pkg.NufftPlan(shape, eps=eps, spread_only=True)
    info = plan.info()
    plan.setpts(torch.from_numpy(k).cuda())
    y = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64)
    grid = torch.empty(shape, dtype=torch.complex64, device="cuda")
    plan.adj(torch.from_numpy(y).cuda(), None, None, grid, 1, 1, 1.0)
    wts = [_axis(k[:, j], shape[j], info["width"], info["beta"]) for j in range(d)]
    sub = "ma,mb,m->ab" if d == 2 else "ma,mb,mc,m->abc"
    ref = np.einsum(sub, *wts, y.astype(np.complex128))
    # the coordinate is rounded to 2^-24 of the period: weights change by beta 1e-7 n
    bound = 2e-6 + 4e-7 * max(shape) * info["beta"]
    assert rel_l2(grid.cpu().numpy(), ref) < bound
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    out = torch.empty(1, M, dtype=torch.complex64, device="cuda")
    plan.op(torch.from_numpy(x).cuda(), None, out, 1, 1, 1.0)
    ref = np.einsum("ma,mb,ab->m" if d == 2 else "ma,mb,mc,abc->m",
                    *wts, x.astype(np.complex128))
    assert rel_l2(out.cpu().numpy()[0], ref) < bound
