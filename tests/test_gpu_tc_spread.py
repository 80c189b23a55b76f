"""The tensor-core spreaders against the per-sample FP32 one.

Plans of two or more transforms with kernel widths up to 7 spread on the tensor
cores (split fp16 operands, fp32 accumulators); ``GBN_SPREAD=gm`` adds every
sample's footprint with FP32 atomics.  Both feed the same transforms, so the
adjoints of the two differ by FP32 rounding: about 1e-6 relative l2 for the
operands' 22 bits, the accumulators' truncation (6e-8 a step, 8 steps) and the
order of the sums; the bound is 5e-6 per transform.

Cases: every width from 2 to 7; odd and even sizes whose last tiles and z
blocks are partial; more samples in one cell than a chunk holds, tiles of one
sample, samples at both ends of the period; transform counts that leave partial
groups (8, 16, 32 per CTA in 2D, 4 in 3D); strengths whose scale differs by
1e12 between transforms and 1e6 inside one.
"""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

BOUND = 5e-6


def _samples(dim, M, rng):
    k = rng.uniform(-0.5, 0.5, (M, dim))
    k[: M // 4] = 0.1234 + rng.uniform(0, 1e-3, (M // 4, dim))  # one cell or two
    k[M // 4: M // 3] *= 0.1
    k[-8:-4] = -0.5
    k[-4:] = np.nextafter(np.float32(0.5), np.float32(0))
    return rng.permutation(k).astype(np.float32)


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("shape,M,C", [((30, 47), 2600, 2), ((251, 16), 3001, 9), ((64, 96), 517, 33),
                                       ((20, 18, 16), 5000, 3), ((9, 41, 25), 2200, 5),
                                       ((33, 12, 70), 130, 2)])
def test_against_fp32_atomics(gpu_pkg, monkeypatch, shape, M, C, eps):
    rng = np.random.default_rng(M + C)
    k = _samples(len(shape), M, rng)
    y = (rng.standard_normal((1, C, M)) + 1j * rng.standard_normal((1, C, M)))
    y *= 10.0 ** rng.uniform(-6, 0, M) * 10.0 ** np.linspace(-6, 6, C)[:, None]
    y = y.astype(np.complex64)
    dens = rng.uniform(0.5, 1.5, M).astype(np.float32)
    out = []
    for spread in ("mma", "gm"):
        monkeypatch.setenv("GBN_SPREAD", spread)
        op = gpu_pkg.MRIGB300(k, shape, n_coils=C, density=dens, squeeze_dims=False, eps=eps)
        out.append(np.asarray(op.adj_op(y)))
    for c in range(C):
        assert rel_l2(out[0][0, c], out[1][0, c]) < BOUND, c


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("shape,M,C", [((30, 47), 2600, 2), ((251, 16), 3001, 17), ((64, 96), 517, 35),
                                       ((250, 256), 900, 66), ((256, 251), 20000, 27),
                                       ((256, 256), 3000, 25), ((20, 18, 16), 5000, 3)])
def test_interp_against_fp32_gather(gpu_pkg, monkeypatch, shape, M, C, eps):
    """The tensor-core interpolation (op, data consistency with density) against
    the per-sample FP32 one, by the same bound; images of scales 1e-6 .. 1e6,
    transform counts that leave partial groups (32, 64 per CTA); sizes and counts
    that keep the FP32 kernels too (other grids than 512^2, up to 24 transforms)."""
    rng = np.random.default_rng(M + C + 1)
    k = _samples(len(shape), M, rng)
    x = rng.standard_normal((1, C, *shape)) + 1j * rng.standard_normal((1, C, *shape))
    x *= 10.0 ** np.linspace(-6, 6, C).reshape(-1, *[1] * len(shape))
    x = x.astype(np.complex64)
    dens = rng.uniform(0.5, 1.5, M).astype(np.float32)
    out = []
    for interp in ("auto", "gm"):
        monkeypatch.setenv("GBN_SPREAD", "mma")
        monkeypatch.setenv("GBN_INTERP", interp)
        op = gpu_pkg.MRIGB300(k, shape, n_coils=C, density=dens, squeeze_dims=False, eps=eps)
        y = np.asarray(op.op(x))
        out.append((y, np.asarray(op.data_consistency(x, 0.25 * y))))
    for c in range(C):
        assert rel_l2(out[0][0][0, c], out[1][0][0, c]) < BOUND, c
        assert rel_l2(out[0][1][0, c], out[1][1][0, c]) < 2 * BOUND, c


@pytest.mark.parametrize("shape,M,C", [((128, 128), 20000, 27), ((128, 128), 16384, 25), ((128, 128), 16383, 25),
                                       ((127, 190), 30000, 48), ((320, 128), 900, 49), ((192, 320), 61440, 33)])
def test_interp_on_other_grids(gpu_pkg, monkeypatch, shape, M, C):
    """The same two on the other grids with fused transforms, on both sides of the
    dispatch's lines: 24 transforms, 48, and a sample for every 4 cells."""
    test_interp_against_fp32_gather(gpu_pkg, monkeypatch, shape, M, C, 1e-6)


@pytest.mark.parametrize("shape,M,C", [((128, 128), 21846, 2), ((128, 128), 21845, 3), ((128, 128), 30000, 5),
                                       ((128, 128), 10923, 9), ((128, 128), 10922, 9), ((100, 90), 36001, 7),
                                       ((9, 130), 4001, 4), ((128, 128), 65536, 25), ((128, 128), 22000, 49)])
def test_interp_from_tiles(gpu_pkg, monkeypatch, shape, M, C):
    """The same two on both sides of the tile kernel's lines (w = 7): samples a cell,
    transforms (groups of 4 and 2 with remainders), grids without fused transforms,
    tiles over both ends of the period, the tensor-core kernel of dense samples."""
    test_interp_against_fp32_gather(gpu_pkg, monkeypatch, shape, M, C, 1e-6)
