"""Plans whose passes grow (``gbn_plan_reserve``) next to what was made before:
batches, captured graphs, Toeplitz embeddings, the memory bound of an operator."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cpx(*s):
    return torch.randn(*s, dtype=torch.complex64, device="cuda")


def _instance(C, n=24, M=300):
    rng = np.random.default_rng(C)
    return {"samples": rng.uniform(-0.5, 0.5, (M, 2)).astype(np.float32), "shape": (n, n), "n_coils": C}


def test_batch_keeps_the_slots_it_was_made_with(gpu_pkg):
    """A batch has as many fine grids for an instance as its plan had transforms
    when the batch was made; binding more coils is refused."""
    from mrinufft_gb300.batched import BatchedNufft

    bat = BatchedNufft([_instance(2), _instance(3)], autotune=False, mode="persistent")
    bat.plans[0].reserve(6)
    bat._bind()  # as many as before
    bat.coils[0] = 3
    with pytest.raises(ValueError):
        bat._bind()


def test_captured_data_consistency_outlives_a_reserve(gpu_pkg):
    """A captured gradient keeps its residual buffer when the plan's passes grow,
    and when a later call with more transforms needs a longer one."""
    C, n, M = 2, 24, 500
    k = torch.from_numpy(np.random.default_rng(1).uniform(-3, 3, (M, 2)).astype(np.float32)).cuda()
    plan = gpu_pkg.NufftPlan((n, n), ntrans=C)
    plan.setpts(k)
    x, y, out = _cpx(C, n, n), _cpx(C, M), _cpx(C, n, n)
    plan.dc(x, y, None, None, out, 1, C, 1.0)
    want = out.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.dc(x, y, None, None, out, 1, C, 1.0)
    plan.reserve(16)
    before = plan.device_bytes
    plan.dc(x, y, None, None, out, 1, C, 1.0)
    assert plan.device_bytes == before  # the same call needs no longer buffer
    x2, y2 = _cpx(16, n, n), _cpx(16, M)
    plan.dc(x2, y2, None, None, torch.empty_like(x2), 1, 16, 1.0)
    assert plan.device_bytes >= before + 8 * 16 * M
    out.zero_()
    graph.replay()
    assert (torch.linalg.norm(out - want) / torch.linalg.norm(want)).item() < 1e-5


def test_corrected_operator_within_the_budget(gpu_pkg, monkeypatch):
    """The off-resonance wrapper raises its operator's passes only within the
    fine-grid budget, old and new grids counted; without device memory for them
    passes stay; the Toeplitz embedding of the operator does not grow."""
    rng = np.random.default_rng(3)
    shape, C, L, M = (32, 24), 4, 9, 400
    k = rng.uniform(-0.5, 0.5, (M, 2)).astype(np.float32)
    tup = _cpx(M, L).cpu().numpy(), _cpx(L, *shape).cpu().numpy()
    smaps = _cpx(C, *shape)

    def make(grids):
        G = 64 * 48
        return gpu_pkg.MRIGB300(k, shape, n_coils=C, smaps=smaps, squeeze_dims=False,
                                fine_budget_bytes=8 * G * grids)

    plain = make(100)
    for grids, want in ((100, 36), (30, 26), (7, 4)):
        op = make(grids)
        held = op.plan.device_bytes
        off = gpu_pkg.MRIFourierCorrectedGB300(op, interpolator=tup)
        assert op.plan.ntrans == want
        assert op.plan.device_bytes - held <= 8 * 64 * 48 * (grids - 4)
        off.compute_interpolator(tup, None, None, None)  # again: no more than the budget
        assert op.plan.device_bytes - held <= 8 * 64 * 48 * (grids - 4)
        assert op._toeplitz().inner_device_bytes() == plain._toeplitz().inner_device_bytes()
    op = make(100)

    def full(n):
        raise MemoryError("no room")

    monkeypatch.setattr(op.plan, "reserve", full)
    off = gpu_pkg.MRIFourierCorrectedGB300(op, interpolator=tup)
    assert op.plan.ntrans == 4
    assert off.op(_cpx(1, 1, *shape)).shape == (1, C, M)
