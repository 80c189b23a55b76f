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
