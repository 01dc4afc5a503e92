"""The 2D trajectory gradient of points in runs and in random order (whose values
are gathered from a point-major copy), with the scratch and without it, against
FP64 autograd (sums of 16 taps x nb entries: 1e-5, as in random order without the
copy), and for the spline, whose windows of width 4 always have 5 taps."""

import ctypes

import pytest
import torch

from conftest import rel_l2
from oracle import interp as OI

from torchlinops_gb300 import _ext, interp

pytestmark = pytest.mark.gpu


def _points(order, n, npts, gen):
    if order == "runs":  # a slow spiral: neighbours in the list are neighbours on the grid
        t = torch.linspace(0, 1, npts)[:, None]
        r = t * (min(n) / 2 - 2.3)
        loc = torch.cat([n[0] / 2 + r * torch.cos(40 * t), n[1] / 2 + r * torch.sin(40 * t)], 1)
    else:
        loc = torch.rand(npts, 2, generator=gen) * torch.tensor(n)
    return torch.floor(loc) + 0.1 + 0.8 * torch.rand(npts, 2, generator=gen)  # clear of the window's edges


@pytest.mark.parametrize("order", ["runs", "random"])
@pytest.mark.parametrize("shape", [(48, 64), (33, 61)])
@pytest.mark.parametrize("nb", [1, 4, 5, 8, 19])
@pytest.mark.parametrize("kernel", ["kaiser_bessel", "spline"])
@pytest.mark.parametrize("scratch", [True, False])
def test_gradient_against_fp64(order, shape, nb, kernel, scratch):
    npts, beta = 3001, OI.nufft_beta(4.0, 1.25)
    gen = torch.Generator().manual_seed(nb + len(order))
    locs = _points(order, shape, npts, gen)
    img = torch.complex(torch.randn(nb, *shape, generator=gen), torch.randn(nb, *shape, generator=gen))
    a = torch.complex(torch.randn(nb, npts, generator=gen), torch.randn(nb, npts, generator=gen))
    kp = dict(beta=beta) if kernel == "kaiser_bessel" else None
    b = beta if kernel == "kaiser_bessel" else 1.0
    ld, im, ad = locs.cuda(), img.cuda(), a.cuda()
    plan = interp.get_plan(ld, shape, 4.0, kernel, "circular", b)
    assert plan.scattered == (order == "random")
    if scratch:
        got = interp._grad_locs(im, ad, ld, 4.0, kernel, 1, "circular", kp)
    else:
        got = torch.empty(npts, 2, device="cuda")
        d = interp._desc(2, shape, (4.0, 4.0), kernel, 1, "circular", b, True, nb, npts)
        assert _ext.lib().tlgb_interp_grad_locs(ctypes.byref(d), ctypes.byref(plan.info), _ext.ptr(plan.buffer), _ext.ptr(ld),
                                                _ext.ptr(im), _ext.ptr(ad), _ext.ptr(got), None, 0,
                                                _ext.stream_ptr(ld.device)) == 0
    ref = OI.grad_locs_interp(img, a, locs, 4.0, kernel=kernel, pad_mode="circular", beta=b)
    assert rel_l2(got.cpu().double(), ref) < 1e-5
