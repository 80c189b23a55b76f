"""2D interpolation of several transforms, w = 7, on both sides of the rule between
tiles and the gather kernel (samples of a subproblem, subproblems, transforms), and the
kernels of one transform and of trajectory gradients on both sides of theirs, against
the per-sample kernel.  Bound as in test_gpu_tc_spread.py."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

BOUND = 5e-6


@pytest.mark.parametrize("C", [2, 4, 9, 20])
@pytest.mark.parametrize("shape,M", [((64, 64), 16000), ((64, 64), 30000), ((64, 64), 48000),
                                     ((128, 120), 24000), ((128, 120), 32000), ((128, 120), 50000)])
def test_tiles_or_gather(gpu_pkg, monkeypatch, shape, M, C):
    rng = np.random.default_rng(M + C)
    k = rng.uniform(-0.5, 0.5, (M, 2)).astype(np.float32)
    x = (rng.standard_normal((1, C, *shape)) + 1j * rng.standard_normal((1, C, *shape))).astype(np.complex64)
    out = []
    for interp in ("auto", "gm"):
        monkeypatch.setenv("GBN_INTERP", interp)
        op = gpu_pkg.MRIGB300(k, shape, n_coils=C, squeeze_dims=False)
        out.append(np.asarray(op.op(x)))
    for c in range(C):
        assert rel_l2(out[0][0, c], out[1][0, c]) < BOUND, c


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("C,M", [(1, 32767), (1, 32768), (2, 65535), (2, 65536), (4, 524288), (3, 40000)])
def test_trajectory_gradient_from_tiles(gpu_pkg, eps, C, M):
    """Trajectory gradients of few transforms (from tiles where there are enough
    samples) against the same transforms beside zeros in a call of eight (from the
    grid).  Rounding of derivative sums, 2e-5 as in test_gpu_widths.py."""
    import torch

    shape = (60, 49)
    g = torch.Generator(device="cuda").manual_seed(M + C)
    cpx = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda", generator=g)
    k = (torch.rand(M, 2, device="cuda", generator=g) - 0.5).cpu().numpy()
    k[:50] = -0.5
    x, dy = cpx(C, *shape), cpx(C, M)
    out = []
    for n in (C, 8):
        op = gpu_pkg.MRIGB300(k, shape, n_coils=n, eps=eps, squeeze_dims=False)
        xn, dn = torch.zeros(n, *shape, dtype=x.dtype, device="cuda"), torch.zeros(n, M, dtype=x.dtype, device="cuda")
        xn[:C], dn[:C] = x, dy
        out.append(op.plan.grad_traj_op(xn, None, dn, torch.empty(M, 2, device="cuda"), 1, n, 1.0).cpu())
    assert rel_l2(out[0], out[1]) < 2e-5


@pytest.mark.parametrize("eps,M", [(1e-3, (1 << 20) - 1), (1e-3, 1 << 20), (1e-4, (1 << 19) - 1), (1e-4, 1 << 19),
                                   (1e-5, (1 << 18) - 1), (1e-5, 1 << 18)])
def test_one_transform_of_many_samples(gpu_pkg, monkeypatch, eps, M):
    rng = np.random.default_rng(M)
    shape = (50, 63)
    k = rng.uniform(-0.5, 0.5, (M, 2)).astype(np.float32)
    x = (rng.standard_normal((1, 1, *shape)) + 1j * rng.standard_normal((1, 1, *shape))).astype(np.complex64)
    out = []
    for interp in ("auto", "gm"):
        monkeypatch.setenv("GBN_INTERP", interp)
        op = gpu_pkg.MRIGB300(k, shape, squeeze_dims=False, eps=eps)
        out.append(np.asarray(op.op(x)))
    assert rel_l2(out[0], out[1]) < BOUND
