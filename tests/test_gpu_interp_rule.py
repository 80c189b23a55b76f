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
