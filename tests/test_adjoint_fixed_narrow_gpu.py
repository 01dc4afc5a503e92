"""tlgb_interp_adjoint_fixed with one entry on a small 2D grid of many points: the
parts of blocks do not fit its buffer, the parts of tiles do. (The sums of 10^4
points per cell differ in their order: 1e-5.)"""

import ctypes

import pytest
import torch

from conftest import rel_l2

import torchlinops_gb300 as T
from torchlinops_gb300 import _ext, interp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,pad", [(6.0, "zero"), (6.0, "circular"), (3.0, "circular")])
def test_parts_of_tiles_where_those_of_blocks_do_not_fit(width, pad):
    n, npts, beta = (64, 61), 1_500_000, T.kaiser_bessel_beta(width, 1.25)
    gen = torch.Generator().manual_seed(1)
    locs = (torch.rand(npts, 2, generator=gen) * torch.tensor(n)).cuda()
    vals = torch.randn(1, npts, dtype=torch.complex64, generator=gen).cuda()
    ref = T.grid(vals, locs, n, width, pad_mode=pad, kernel_params=dict(beta=beta))
    plan = interp.get_plan(locs, n, width, "kaiser_bessel", pad, beta)
    assert plan.info.n_blk_partials * 64 * 16 * 4 > 32 << 20
    desc = interp._desc(2, n, (width,) * 2, "kaiser_bessel", 1, pad, beta, True, 1, npts)
    L = _ext.lib()
    for _ in range(2):
        out = torch.full((1, *n), float("nan"), dtype=torch.complex64, device="cuda")
        st = L.tlgb_interp_adjoint_fixed(ctypes.byref(desc), ctypes.byref(plan.info), _ext.ptr(plan.buffer), _ext.ptr(locs),
                                         _ext.ptr(torch.view_as_real(vals)), _ext.ptr(torch.view_as_real(out)),
                                         _ext.stream_ptr(out.device))
        assert st == _ext.TLGB_OK, L.tlgb_last_error()
        assert rel_l2(out.cpu(), ref.cpu()) < 1e-5
