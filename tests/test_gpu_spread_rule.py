"""Plans of several transforms spread on the tensor cores only where the samples pay
for it; the others take FP32 kernels on the same tiles and columns.  Against the
per-sample FP32 atomics on both sides of the rule: few and many samples, few and many
transforms, clusters that fill a column's chunk, every width, odd grids.

Bound: FP32 rounding and the order of sums, 5e-6 relative l2 per transform (see
test_gpu_tc_spread.py)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

BOUND = 5e-6


def _check(gpu_pkg, monkeypatch, k, shape, C, eps, M, one=False):
    rng = np.random.default_rng(M + C)
    y = (rng.standard_normal((1, C, M)) + 1j * rng.standard_normal((1, C, M))).astype(np.complex64)
    dens = rng.uniform(0.5, 1.5, M).astype(np.float32)
    out = []
    for spread in (None, "gm"):
        monkeypatch.delenv("GBN_SPREAD", raising=False)
        if spread:
            monkeypatch.setenv("GBN_SPREAD", spread)
        op = gpu_pkg.MRIGB300(k, shape, n_coils=C, density=dens, squeeze_dims=False, eps=eps)
        out.append([np.asarray(op.adj_op(y)[0, c]) for c in range(C)])
        if one:  # one transform on the plan of several
            out[-1].append(np.asarray(op._adj_op(y[0, :1], None))[0])
    for c, (a, b) in enumerate(zip(*out)):
        assert rel_l2(a, b) < BOUND, c


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("shape,M,C", [((20, 18, 16), 5000, 3), ((9, 41, 25), 2200, 9), ((33, 12, 70), 130, 2),
                                       ((24, 24, 24), 1, 4), ((30, 47), 2600, 2), ((251, 16), 300, 9),
                                       ((64, 96), 517, 33)])
def test_few_samples(gpu_pkg, monkeypatch, shape, M, C, eps):
    rng = np.random.default_rng(M)
    k = rng.uniform(-0.5, 0.5, (M, len(shape)))
    k[: M // 3] = 0.1234 + rng.uniform(0, 1e-3, (M // 3, len(shape)))  # more than a chunk in one column
    k[-(M // 9):] = -0.5
    _check(gpu_pkg, monkeypatch, rng.permutation(k).astype(np.float32), shape, C, eps, M, one=True)


@pytest.mark.parametrize("M", [32767, 32768, 60000])
@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 7, 8])
def test_both_sides_in_3d(gpu_pkg, monkeypatch, M, C):
    """28 x 30 x 26 voxels: a is about 17 for 32 768 samples, 30 for 60 000 (lines at
    1.3, 2, 3, 12 and 32)."""
    rng = np.random.default_rng(M + C)
    k = rng.uniform(-0.5, 0.5, (M, 3)).astype(np.float32)
    _check(gpu_pkg, monkeypatch, k, (28, 30, 26), C, 1e-6, M, one=True)
    _check(gpu_pkg, monkeypatch, k, (64, 60, 64), C, 1e-3, M)


@pytest.mark.parametrize("M", [2000, 9000, 40000])
@pytest.mark.parametrize("C", [2, 4, 8, 16, 17, 40])
def test_both_sides_in_2d(gpu_pkg, monkeypatch, M, C):
    rng = np.random.default_rng(M + C)
    k = rng.uniform(-0.5, 0.5, (M, 2)).astype(np.float32)
    _check(gpu_pkg, monkeypatch, k, (110, 128), C, 1e-6, M)
    _check(gpu_pkg, monkeypatch, k, (110, 128), C, 1e-4, M)
