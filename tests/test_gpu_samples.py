"""``samples`` of an operator: Fortran-ordered float32 radians, as they were set."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_samples_are_those_that_were_set(gpu_pkg, dim):
    rng = np.random.default_rng(dim)
    shape = (16, 12, 14)[:dim]
    k = torch.from_numpy(rng.uniform(-3, 3, (257, dim)).astype(np.float32)).cuda()
    want = k.cpu().numpy()
    op = gpu_pkg.MRIGB300(k, shape)
    k.zero_()  # the caller's array is its own
    got = op.samples
    assert got.flags.f_contiguous and got.dtype == np.float32 and got.shape == want.shape
    np.testing.assert_array_equal(got, want)
    assert op.samples is got
    new = rng.uniform(-3, 3, (100, dim)).astype(np.float32)
    op.update_samples(new)
    np.testing.assert_array_equal(op.samples, new)


def test_samples_are_copied_when_they_are_set(gpu_pkg, monkeypatch):
    """Reading ``samples`` neither copies nor waits, so that it is possible inside a
    stream capture; after an update that fails they are those that were set."""
    rng = np.random.default_rng(9)
    k = rng.uniform(-3, 3, (300, 2)).astype(np.float32)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        op = gpu_pkg.MRIGB300(torch.from_numpy(k).cuda(), (16, 12))
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1
        got = op.samples
    np.testing.assert_array_equal(got, k)
    new = rng.uniform(-3, 3, (100, 2)).astype(np.float32)

    def refuse(samples):
        raise MemoryError("no room for the points")

    monkeypatch.setattr(op.plan, "setpts", refuse)
    with pytest.raises(MemoryError):
        op.update_samples(new)
    np.testing.assert_array_equal(op.samples, new)
    assert op.n_samples == 100
