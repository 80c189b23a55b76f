"""Pipe density iterations on real grids against the complex kernels.

Same weights and sums, on floats: every term is positive, so the two differ by the
rounding of the sums (up to 512 terms before a flush, 6e-8 each at random signs:
about 1.4e-6) in spread and interp of each iteration, and a division passes errors
on at about their size; three iterations stay below 2e-5 relative.

Cases: widths 4 to 7 and 3 (complex kernels only), odd cell counts, axes shorter
than the z window, one sample, clusters that fill several chunks, the ends of the
period, partial tiles; 2D plans keep the complex kernels.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points(dim, M, rng):
    k = rng.uniform(-np.pi, np.pi, (M, dim))
    k[: M // 3] = 0.3 + rng.uniform(0, 1e-2, (M // 3, dim))
    k[M // 3: M // 2] *= 0.1
    k[: min(M, 2)] = -np.pi
    return torch.as_tensor(rng.permutation(k).astype(np.float32), device="cuda")


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("shape,M", [((32, 32, 32), 20000), ((9, 13, 11), 1), ((9, 11, 5), 700),
                                     ((33, 40, 17), 3001), ((8, 8, 64), 129), ((17, 30), 500)])
def test_real_equals_complex(gpu_pkg, shape, M, eps):
    rng = np.random.default_rng(M)
    plan = gpu_pkg.plan.NufftPlan(shape, eps=eps, ntrans=1, spread_only=True)
    assert plan.real_pipe == (len(shape) == 3 and eps < 1e-2)
    plan.setpts(_points(len(shape), M, rng))
    w = torch.as_tensor(rng.uniform(0.5, 2, M).astype(np.float32), device="cuda")
    if not plan.real_pipe:
        with pytest.raises(ValueError):
            plan.pipe(w, 1, 1.0)
        return
    ref = plan.pipe(w.to(torch.complex64), 3, 0.25)
    out = plan.pipe(w.clone(), 3, 0.25)
    assert not ref.imag.any()
    torch.testing.assert_close(out, ref.real, rtol=2e-5, atol=0)


def test_other_kernels_keep_complex(gpu_pkg, monkeypatch):
    for name, value in (("GBN_SPREAD", "gm"), ("GBN_SPREAD", "stream"), ("GBN_INTERP", "wc"), ("GBN_BINS3", "6,8,8")):
        with monkeypatch.context() as m:
            m.setenv(name, value)
            assert not gpu_pkg.plan.NufftPlan((32, 32, 32), ntrans=1, spread_only=True).real_pipe


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("eps,shape", [(1e-6, (24, 20, 28)), (1e-6, (20, 24, 27)), (1e-5, (13, 22, 40)),
                                       (1e-4, (24, 8, 64)), (1e-3, (9, 10, 12))])
def test_tile_copies(gpu_pkg, monkeypatch, eps, shape, offset):
    """Interpolation from a caller's 3D grid: tiles copied two cells at a time (even
    grids that start on a pair) or one (odd ones, grids one cell off), with tiles
    over both ends of the period, against the direct FP32 kernel; sums of the same
    terms in another order: 343 of them, 2e-6 of the largest value."""
    rng = np.random.default_rng(7)
    M = 3000
    pts = _points(3, M, rng)
    buf = torch.as_tensor(rng.standard_normal(2 * (2 * int(np.prod(shape)) + 2)).astype(np.float32), device="cuda")
    x = torch.view_as_complex(buf.reshape(-1, 2))[offset: offset + 2 * int(np.prod(shape))].reshape(2, *shape)
    out = []
    for interp in ("auto", "gm"):
        monkeypatch.setenv("GBN_INTERP", interp)
        plan = gpu_pkg.plan.NufftPlan(shape, eps=eps, ntrans=2, spread_only=True)
        plan.setpts(pts)
        y = torch.empty((2, M), dtype=torch.complex64, device="cuda")
        plan.op(x, None, y, 1, 2, 1.0)
        out.append(y)
    assert (out[0] - out[1]).abs().max() < 2e-6 * out[1].abs().max()
