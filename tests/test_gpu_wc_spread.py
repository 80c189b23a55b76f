"""2D spreading of widths 4 to 7 by eight lanes a sample, and its rule against the
per-sample atomics, which it has to equal to the rounding of sums (5e-6, see
test_gpu_tc_spread.py): odd grids, both ends of the period, last warps that are not
full, both sides of half a million samples and of the densities."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("shape,M,C", [((17, 30), 1, 1), ((30, 47), 2601, 1), ((64, 50), 5003, 3),
                                       ((80, 64), (1 << 19) - 1, 1), ((80, 64), 1 << 19, 1),
                                       ((400, 410), 1 << 19, 1), ((50, 60), 1 << 19, 1)])
def test_against_per_sample_atomics(gpu_pkg, monkeypatch, shape, M, C, eps):
    rng = np.random.default_rng(M + C)
    k = rng.uniform(-0.5, 0.5, (M, 2))
    k[: M // 50] = -0.5
    k = k.astype(np.float32)
    y = (rng.standard_normal((1, C, M)) + 1j * rng.standard_normal((1, C, M))).astype(np.complex64)
    dens = rng.uniform(0.5, 1.5, M).astype(np.float32)
    out = []
    for spread in (None, "gm"):
        monkeypatch.delenv("GBN_SPREAD", raising=False)
        if spread:
            monkeypatch.setenv("GBN_SPREAD", spread)
        op = gpu_pkg.MRIGB300(k, shape, n_coils=C, density=dens, squeeze_dims=False, eps=eps)
        out.append(np.asarray(op.adj_op(y)))
    for c in range(C):
        assert rel_l2(out[0][0, c], out[1][0, c]) < 5e-6, c
