"""The 2D trajectory gradient on the gather's ring at the sizes where it can go
wrong, against FP64 autograd: batches below and above a group of 8 entries and
in several runs, items of a few and of many points, odd grids (plain region
copies), wraps, and kernels narrower than the record."""

import pytest
import torch

from conftest import rel_l2
from oracle import interp as OI

import torchlinops_gb300 as T

pytestmark = pytest.mark.gpu
# FP32 sums of 16 taps x nb entries against FP64: 8e-7 expected at nb = 40 (sqrt(640) roundings of 6e-8 against
# a sum that grows alike, three steps of them); the derivative of a weight 0.1 from the window's edge adds 1e-6.
TOL = 1e-5


@pytest.mark.parametrize("shape,npts", [((48, 40), 2500), ((33, 61), 1500), ((17, 13), 700), ((9, 10), 1), ((40, 64), 33)])
@pytest.mark.parametrize("width,pad", [(4.0, "circular"), (4.0, "zero"), (3.0, "zero"), (2.0, "circular")])
@pytest.mark.parametrize("nb", [1, 3, 9, 40])
def test_gradient_against_fp64(shape, npts, width, pad, nb):
    gen = torch.Generator().manual_seed(npts + nb)
    n = torch.tensor(shape, dtype=torch.float32)
    lo = torch.floor(torch.rand(npts, 2, generator=gen) * (n + 2)) - 1
    lo[: npts // 2] = torch.floor(n / 3) + torch.floor(torch.rand(npts // 2, 2, generator=gen) * 5)
    locs = lo + 0.1 + 0.8 * torch.rand(npts, 2, generator=gen) - (width / 2) % 1.0  # clear of the window's edges
    img = torch.complex(torch.randn(nb, *shape, generator=gen), torch.randn(nb, *shape, generator=gen))
    a = torch.complex(torch.randn(nb, npts, generator=gen), torch.randn(nb, npts, generator=gen))
    beta = OI.nufft_beta(width, 1.25)
    L = locs.to("cuda").requires_grad_(True)
    out = T.interpolate(img.to("cuda"), L, width, pad_mode=pad, kernel_params=dict(beta=beta))
    (a.to("cuda").conj() * out).real.sum().backward()
    ref = OI.grad_locs_interp(img, a, locs, width, pad_mode=pad, beta=beta)
    assert rel_l2(L.grad.cpu(), ref) < TOL
