"""Gridding on block lists where a window can meet three blocks along a
dimension (circular grids whose last block is a partial one, windows of more
than 5 taps in 3D), where the kernel is wider or narrower than the NUFFT's,
and on the smallest grids that have block lists: against the CPU oracle, the
lists bit for bit."""

import numpy as np
import pytest
import torch

from oracle import binning as OB
from oracle import interp as OI
from conftest import rel_l2

import torchlinops_gb300 as T
from torchlinops_gb300 import interp

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-5

# (grid, width, pad, rows per dim in the lists)
CASES = [
    ((25, 30, 27), 4.0, "circular", 3),
    ((8, 9, 11), 4.0, "circular", 3),  # the smallest grids with 8-cell tiles
    ((41, 24, 26), 4.0, "circular", 3),
    ((33, 49), 4.0, "circular", 3),
    ((16, 23), 4.0, "circular", 2),
    ((24, 28, 32), 3.0, "circular", 2),
    ((24, 30, 29), 6.0, "zero", 3),
    ((28, 24, 32), 6.0, "circular", 3),
    ((20, 33, 26), 8.0, "zero", 3),
    ((40, 61), 6.0, "zero", 2),
    ((48, 50), 6.0, "circular", 3),
    ((64, 40), 8.0, "circular", 2),
]


def _locs(shape, gen):
    n = torch.tensor(shape, dtype=torch.float32)
    spread = torch.rand(6000, len(shape), generator=gen) * (n + 6) - 3  # past both edges
    dense = n - 0.5 + torch.rand(2000, len(shape), generator=gen)  # around the wrap, split blocks
    ints = torch.randint(-2, min(shape) + 2, (200, len(shape)), generator=gen).float()
    return torch.cat([spread, dense, ints])


@pytest.mark.parametrize("shape,width,pad,rows", CASES)
@pytest.mark.parametrize("nb", [1, 3, 8, 11])
def test_block_gridding_against_oracle(shape, width, pad, rows, nb):
    gen = torch.Generator().manual_seed(nb + sum(shape))
    locs = _locs(shape, gen)
    pts = torch.complex(torch.randn(nb, len(locs), generator=gen), torch.randn(nb, len(locs), generator=gen))
    beta = OI.nufft_beta(width, 1.25)
    kw = dict(kernel="spline" if nb == 3 else "kaiser_bessel", pad_mode=pad)
    got = T.grid(pts.to(DEV), locs.to(DEV), shape, width, kernel_params=dict(beta=beta), **kw)
    again = T.grid(pts.to(DEV), locs.to(DEV), shape, width, kernel_params=dict(beta=beta), **kw)
    assert torch.equal(got, again)
    assert rel_l2(got.cpu(), OI.grid(pts, locs, shape, width, beta=beta, **kw)) < TOL
    assert rel_l2(got.cpu(), OI.grid(pts, locs, shape, width, beta=beta, dtype=torch.float64, **kw)) < TOL


@pytest.mark.parametrize("shape,width,pad,rows", CASES)
def test_block_lists_of_three_rows(shape, width, pad, rows):
    gen = torch.Generator().manual_seed(sum(shape))
    locs = _locs(shape, gen)
    locs[:9, 0] = float("nan")
    keys, pts = OB.block_pairs(locs, shape, width, "kaiser_bessel", pad)
    plan = interp.InterpolatePlan(locs.to(DEV), shape, width, "kaiser_bessel", pad, 7.0)
    info = plan.info
    off, n = int(info.off_blk_entries), int(info.n_blk_entries)
    assert n == len(pts)
    got = plan.buffer[off:off + 4 * n].view(torch.int32).cpu().numpy().astype(np.int64) & 0xFFFFFFFF
    # the oracle holds the blocks' indices per dim as 3 x 1 bit above the point
    # (they run to 2 here, so it cannot tell them apart): compare the points,
    # whose blocks are fixed by the order of the list
    shift = 27 if rows == 3 else 29
    npt = len(locs)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(got & ((1 << shift) - 1), (pts & ((1 << 29) - 1))[order]) and npt < 1 << 27


def test_non_finite_values_stay_in_their_windows_across_a_partial_block():
    shape, width = (25, 30, 27), 4.0
    gen = torch.Generator().manual_seed(3)
    locs = _locs(shape, gen)[:500]
    locs[0] = torch.tensor([24.3, 29.1, 26.7])  # wraps along every dim
    pts = torch.complex(torch.randn(2, 500, generator=gen), torch.randn(2, 500, generator=gen))
    bad = pts.clone()
    bad[0, 0] = complex(float("nan"), 1.0)
    kp = dict(beta=OI.nufft_beta(width, 1.25))
    good = T.grid(pts.to(DEV), locs.to(DEV), shape, width, kernel_params=kp).cpu()
    got = T.grid(bad.to(DEV), locs.to(DEV), shape, width, kernel_params=kp).cpu()
    hit = torch.zeros(shape, dtype=torch.bool)
    ax = [[int(v) % n for v in range(int(np.ceil(x - 2)), int(np.floor(x + 2)) + 1)] for x, n in zip(locs[0].tolist(), shape)]
    hit[np.ix_(*ax)] = True
    assert bool(got[0][hit].isnan().all()) and not bool(got[0][~hit].isnan().any())
    assert rel_l2(got[0][~hit], good[0][~hit]) < TOL and rel_l2(got[1], good[1]) < TOL
