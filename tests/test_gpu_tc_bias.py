"""What the tensor-core interpolation gives back for the truncation of its accumulators
follows the width: half of the w rows, 6e-8 each.  The loss of a row depends on how the
cells cancel, so the mean against the FP32 kernel, <a, b> / <b, b> - 1, may be half of
that off."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
def test_mean_against_fp32(gpu_pkg, monkeypatch, eps):
    g = torch.Generator(device="cuda").manual_seed(1)
    shape, C, M = (256, 256), 64, 100000
    k = (torch.rand(M, 2, device="cuda", generator=g) - 0.5) * 6.28
    x = torch.randn(C, *shape, dtype=torch.complex64, device="cuda", generator=g)
    monkeypatch.setenv("GBN_SPREAD", "mma")
    out = []
    for interp in ("auto", "gm"):
        monkeypatch.setenv("GBN_INTERP", interp)
        plan = gpu_pkg.NufftPlan(shape, ntrans=C, eps=eps)
        plan.setpts(k)
        y = plan.op(x, None, torch.empty(C, M, dtype=torch.complex64, device="cuda"), 1, C, 1.0)
        out.append(y.to(torch.complex128).flatten())
    bias = (torch.vdot(out[1], out[0]) / torch.vdot(out[1], out[1])).real.item() - 1
    assert abs(bias) < 0.5 * 0.5 * plan.info()["width"] * 6e-8
