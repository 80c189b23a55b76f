"""How a tensor-core wait that ran out is reported.  No kernel is made to wait: the
word that it would set is set on the host."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _word(plan):
    p = ctypes.POINTER(ctypes.c_int)()
    assert plan.lib.gbn_plan_error_word(plan._h, ctypes.byref(p)) == 0
    return p


def _op(pkg, C, seed=0):
    k = np.random.default_rng(seed).uniform(-0.5, 0.5, (400, 2)).astype(np.float32)
    return pkg.MRIGB300(k, (24, 20), n_coils=C, squeeze_dims=False)


def _error(pkg):
    from mrinufft_gb300 import _lib

    return _lib.GB300Error


def test_reported_once_and_for_its_plan_alone(gpu_pkg):
    a, b, one = _op(gpu_pkg, 3), _op(gpu_pkg, 3, 1), _op(gpu_pkg, 1)
    y = torch.randn(1, 3, 400, dtype=torch.complex64, device="cuda")
    want = a.adj_op(y)
    assert not _word(one.plan)  # a plan of one transform has no such kernels
    _word(a.plan)[0] = 1
    b.adj_op(y)
    b.plan.check()
    with pytest.raises(_error(gpu_pkg)):
        a.adj_op(y)
    assert torch.linalg.norm(a.adj_op(y) - want) < 1e-5 * torch.linalg.norm(want)
    _word(a.plan)[0] = 1
    with pytest.raises(_error(gpu_pkg)):
        a.plan.check()
    a.plan.check()


def test_host_results_are_checked_by_their_own_call(gpu_pkg, monkeypatch):
    from mrinufft_gb300 import _array

    op = _op(gpu_pkg, 3)
    plain = _array.from_tensor

    def gave_up(t, like):  # as if a kernel of this call had
        _word(op.plan)[0] = 1
        return plain(t, like)

    y = np.ones((1, 3, 400), np.complex64)
    x = op.adj_op(y)
    monkeypatch.setattr(_array, "from_tensor", gave_up)
    for call in (lambda: op.adj_op(y), lambda: op.op(x), lambda: op.data_consistency(x, y),
                 lambda: op.adj_op(torch.from_numpy(y))):
        with pytest.raises(_error(gpu_pkg)):
            call()


def test_replays_are_checked(gpu_pkg):
    from mrinufft_gb300.batched import BatchedNufft

    k = np.random.default_rng(2).uniform(-0.5, 0.5, (300, 2)).astype(np.float32)
    bat = BatchedNufft([{"samples": k, "shape": (24, 24), "n_coils": 3}], autotune=False)
    bat.replay()
    torch.cuda.synchronize()
    bat.check()
    _word(bat.plans[0])[0] = 1
    with pytest.raises(_error(gpu_pkg)):
        bat.replay()
    bat.replay()


def test_words_of_more_plans_than_a_page(gpu_pkg):
    """Every living plan has a word of its own; words come back with their plans."""
    plans = [gpu_pkg.NufftPlan((4, 4), ntrans=2) for _ in range(1030)]
    words = {ctypes.addressof(_word(p).contents) for p in plans}
    assert len(words) == len(plans)
    _word(plans[7])[0] = 1
    plans = None  # noqa: F841
    again = [gpu_pkg.NufftPlan((4, 4), ntrans=2) for _ in range(1030)]
    for p in again:
        p.check()
