"""Gridding from the block lists where the chunk stream can go wrong: lists of a
few entries and of many chunks, runs of empty blocks, several groups of entries
in one launch, values read with and without their transposition, and NaN or
Inf among the values, which reach the cells of their point's window and no other."""

import pytest
import torch

from conftest import rel_l2
from oracle import interp as OI

import torchlinops_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,npts", [((20, 17, 30), 15), ((32, 32, 32), 33), ((24, 28, 20), 6000), ((64, 70), 17), ((50, 33), 5000)])
@pytest.mark.parametrize("nb", [1, 2, 3, 8, 21])
@pytest.mark.parametrize("bad", [None, float("nan"), float("inf")])
def test_gridding_against_oracle(shape, npts, nb, bad):
    gen = torch.Generator().manual_seed(npts + nb)
    n = torch.tensor(shape, dtype=torch.float32)
    locs = torch.rand(npts, len(shape), generator=gen) * n
    locs[: npts // 2] = n / 3 + torch.rand(npts // 2, len(shape), generator=gen) * 4  # dense blocks next to empty ones
    vals = torch.complex(torch.randn(nb, npts, generator=gen), torch.randn(nb, npts, generator=gen))
    beta = OI.nufft_beta(4.0, 1.25)
    want = OI.grid(vals, locs, shape, 4.0, beta=beta)
    hit = torch.zeros(shape, dtype=torch.bool)
    if bad is not None:
        one = torch.zeros(1, npts, dtype=torch.complex64)
        one[0, npts - 1] = 1.0
        hit = OI.grid(one, locs, shape, 4.0, beta=beta)[0].abs() > 0
        vals[nb - 1, npts - 1] = bad
    got = T.grid(vals.cuda(), locs.cuda(), shape, 4.0, kernel_params=dict(beta=beta)).cpu()
    if bad is not None:
        assert not bool(torch.isfinite(torch.view_as_real(got[nb - 1])).all(-1)[hit].any())
        got[nb - 1][hit] = 0
        want[nb - 1][hit] = 0
    assert bool(torch.isfinite(torch.view_as_real(got)).all())
    assert rel_l2(got, want) < 1e-5
