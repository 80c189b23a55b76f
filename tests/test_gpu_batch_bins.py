"""Bins of batches: the tuner times the plan's own choice too, persistent batches have
tiles for the row spreader."""

import json

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _instances(dim):
    rng = np.random.default_rng(dim)
    out = []
    for n, C, M in ((24, 4, 900), (20, 1, 400)):
        maps = rng.standard_normal((C, *(n,) * dim)) + 1j * rng.standard_normal((C, *(n,) * dim))
        out.append({"samples": rng.uniform(-0.5, 0.5, (M, dim)).astype(np.float32), "shape": (n,) * dim,
                    "smaps": maps.astype(np.complex64)})
    return out


@pytest.mark.parametrize("dim", [2, 3])
def test_own_bins_are_a_candidate(gpu_pkg, tmp_path, dim):
    from mrinufft_gb300.autotune import OWN, Autotuner
    from mrinufft_gb300.batched import BatchedNufft

    path = tmp_path / "tune.json"
    BatchedNufft(_instances(dim), tuner=Autotuner(cache_path=path, interp_methods=("auto",)))
    for c in json.loads(path.read_text()).values():
        assert f"{OWN['bins']}/auto" in c["timings"] and c["ms"] == min(c["timings"].values())
    # a stored choice of the plan's own bins, and one made before it was a candidate
    tuner = Autotuner(cache_path=path, interp_methods=("auto",))
    key = next(iter(tuner.cache))
    tuner.cache = {k: {"bins": None, "interp": "auto", "maxsub": 512} for k in tuner.cache}
    own = BatchedNufft(_instances(dim), tuner=tuner)
    plain = BatchedNufft(_instances(dim), autotune=False)
    assert [p.info()["bins"] for p in own.plans] == [p.info()["bins"] for p in plain.plans]
    assert key.endswith("+own") and Autotuner(own=False, interp_methods=("auto",)).key((8, 8), 9, 1)[-4:] == "auto"


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("autotune", [False, True])
def test_persistent_bins(gpu_pkg, monkeypatch, tmp_path, dim, autotune):
    from mrinufft_gb300.batched import BatchedNufft

    monkeypatch.setenv("GBN_TUNE_CACHE", str(tmp_path / "t.json"))
    insts = _instances(dim)
    bat = BatchedNufft(insts, autotune=autotune, mode="persistent")
    if dim == 3:  # tiles of at most 16 rows an axis: bins of up to 9
        assert all(max(p.info()["bins"]) <= 9 for p in bat.plans)
    y = [torch.randn(k.shape, dtype=torch.complex64, device="cuda") for k in bat.ksps]
    bat.set_kspace(y)
    for inst, yi, x in zip(insts, y, bat.adj()):
        op = gpu_pkg.MRIGB300(inst["samples"], inst["shape"], n_coils=len(inst["smaps"]), smaps=inst["smaps"],
                              squeeze_dims=False)
        assert rel_l2(x.cpu().numpy(), op.adj_op(yi[None]).cpu().numpy()) < 1e-5
