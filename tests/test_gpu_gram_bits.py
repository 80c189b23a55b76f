"""The Toeplitz Gram has no atomics: repeated calls give the same bits, on the 2D
grids with fused transforms (square, uneven, one coil, several passes) as on others."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,C", [((128, 128), 16), ((192, 192), 5), ((256, 256), 16), ((320, 128), 7),
                                     ((384, 384), 12), ((100, 250), 16), ((128, 128), 70), ((128, 128), 1),
                                     ((90, 100), 8), ((64, 64, 64), 6)])
def test_same_bits_every_time(gpu_pkg, shape, C):
    rng = np.random.default_rng(C)
    k = rng.uniform(-0.5, 0.5, (3000, len(shape))).astype(np.float32)
    cpx = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda")
    op = gpu_pkg.MRIGB300(k, shape, n_coils=C, smaps=cpx(C, *shape), squeeze_dims=False)
    x = cpx(1, 1, *shape)
    want = op.gram_op(x)
    ref = op.adj_op(op.op(x))
    assert torch.linalg.norm(want - ref) < 2e-5 * torch.linalg.norm(ref)
    for _ in range(8):
        assert torch.equal(op.gram_op(x), want)
