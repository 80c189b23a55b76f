"""The z transforms of stacks, one kernel or three passes as the rule has it: against
torch's FFT in double precision, on both sides of it (planes and their factors, few and
many columns, with and without maps, a subset of the planes).

Bound: sums of up to 126 terms in FP32, 1e-6 relative l2 (sqrt(126) * 6e-8 = 7e-7)."""

import ctypes

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [9, 25, 45, 64, 65, 70, 75, 90, 100, 120, 126])
@pytest.mark.parametrize("xy,C", [((9, 7), 1), ((9, 7), 5), ((97, 130), 2), ((160, 150), 4)])
def test_z_transforms(gpu_pkg, xy, C, nz):
    g = torch.Generator(device="cuda").manual_seed(nz)
    cpx = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda", generator=g)
    shape = (*xy, nz)
    k2 = np.zeros((4, 2), np.float32)
    for zi in (np.arange(nz), np.arange(0, nz, 4)):
        op = gpu_pkg.MRIStackedGB300(k2, shape, n_coils=C, z_index=zi)
        ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
        keep = torch.from_numpy(zi).cuda()
        for maps in (None, cpx(C, *shape)):
            img = cpx(1 if maps is not None else C, *shape)
            planes = torch.empty(C, len(zi), *xy, dtype=torch.complex64, device="cuda")
            assert op.lib.gbn_stack_fwd(op._stack, ptr(img), ptr(maps), ptr(planes), C, op._st()) == 0
            v = img.to(torch.complex128) * (1 if maps is None else maps.to(torch.complex128))
            f = torch.fft.fftshift(torch.fft.fft(torch.fft.ifftshift(v, dim=3), dim=3), dim=3) / np.sqrt(2 * nz)
            ref = f[..., keep].permute(0, 3, 1, 2)
            assert rel_l2(planes.cpu(), ref.cpu()) < 1e-6
            back = cpx(*img.shape)
            start = back.to(torch.complex128)
            for accumulate in (0, 1):
                assert op.lib.gbn_stack_adj(op._stack, ptr(planes), ptr(maps), ptr(back), C, accumulate, op._st()) == 0
                full = torch.zeros(C, *shape, dtype=torch.complex128, device="cuda")
                full[..., keep] = planes.to(torch.complex128).permute(0, 2, 3, 1)
                b = torch.fft.fftshift(torch.fft.ifft(torch.fft.ifftshift(full, dim=3), dim=3), dim=3) * nz / np.sqrt(2 * nz)
                if maps is not None:
                    b = (b * maps.to(torch.complex128).conj()).sum(0, keepdim=True)
                want = b + (start if accumulate else 0)
                assert rel_l2(back.cpu(), want.cpu()) < 1e-6
                start = want
