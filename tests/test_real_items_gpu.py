"""Ungridding of real values where a CTA takes several items, of one tile and of
neighbouring ones, with remainders: against the complex values' kernel, whose
results the oracle pins (float32 sums of the same taps in another order, weights
equal to some ulps: 5e-6)."""

import pytest
import torch

from conftest import rel_l2

import torchlinops_gb300 as T
from torchlinops_gb300 import interp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,npts,nb,width", [((17, 16, 24), 200_000, 3, 4.0), ((24, 24, 25), 330_000, 8, 3.0),
                                                 ((40, 50), 230_000, 24, 4.0), ((33, 64), 200_000, 31, 6.0),
                                                 ((16, 16), 700_000, 1, 8.0), ((40, 50), 300, 2, 4.0)])
def test_real_against_complex(shape, npts, nb, width):
    gen = torch.Generator().manual_seed(npts)
    n = torch.tensor(shape, dtype=torch.float32)
    locs = torch.rand(npts, len(shape), generator=gen) * n
    locs[: npts // 3] = n / 2 + torch.rand(npts // 3, len(shape), generator=gen) * 4  # tiles of many items beside lighter ones
    img = torch.randn(nb, *shape, generator=gen).cuda()
    locs = locs.cuda()
    kp = dict(beta=T.kaiser_bessel_beta(width, 1.25))
    got = T.ungrid(img, locs, width, kernel_params=kp)
    want = T.ungrid(img.to(torch.complex64), locs, width, kernel_params=kp).real
    assert rel_l2(got.cpu(), want.cpu()) < 5e-6
    assert interp.get_plan(locs, shape, width, "kaiser_bessel", "circular", kp["beta"]).info.n_fwd_items >= 1
