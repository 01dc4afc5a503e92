"""The 2D trajectory gradient into memory that is only 4-byte aligned (a C caller's
packed buffer), against the aligned result: other kernels, FP32 sums of 16 taps x
nb entries (1e-5)."""

import ctypes

import pytest
import torch

from conftest import rel_l2

import torchlinops_gb300 as T
from torchlinops_gb300 import _ext, interp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 9])
def test_gradient_at_an_odd_float(nb):
    n, npts, beta = (40, 48), 3000, T.kaiser_bessel_beta(4.0, 1.25)
    gen = torch.Generator().manual_seed(nb)
    locs = (torch.rand(npts, 2, generator=gen) * torch.tensor(n)).cuda()
    img = torch.randn(nb, *n, dtype=torch.complex64, generator=gen).cuda()
    a = torch.randn(nb, npts, dtype=torch.complex64, generator=gen).cuda()
    want = interp._grad_locs(img, a, locs, 4.0, "kaiser_bessel", 1, "circular", dict(beta=beta))
    plan = interp.get_plan(locs, n, 4.0, "kaiser_bessel", "circular", beta)
    desc = interp._desc(2, n, (4.0,) * 2, "kaiser_bessel", 1, "circular", beta, True, nb, npts)
    buf = torch.full((2 * npts + 2,), -7.0, device="cuda")
    out = buf[1:-1]
    assert out.data_ptr() % 8 == 4
    st = _ext.lib().tlgb_interp_grad_locs(ctypes.byref(desc), ctypes.byref(plan.info), _ext.ptr(plan.buffer), _ext.ptr(locs),
                                          _ext.ptr(torch.view_as_real(img)), _ext.ptr(torch.view_as_real(a)), _ext.ptr(out),
                                          None, 0, _ext.stream_ptr(out.device))
    assert st == _ext.TLGB_OK, _ext.lib().tlgb_last_error()
    assert rel_l2(out.view(npts, 2).cpu(), want.cpu()) < 1e-5
    assert float(buf[0]) == -7.0 and float(buf[-1]) == -7.0
