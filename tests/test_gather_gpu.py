"""The ring-buffered gather at the sizes where it can go wrong, against the CPU
oracle: items of one point up to several items of a tile, every group size and
partial groups, regions copied by TMA and by plain copies (odd rows, wraps,
grids barely larger than a region), windows of more taps than a record holds,
wide and narrow kernels, and results that go through the items' order."""

import pytest
import torch

from conftest import rel_l2
from oracle import interp as OI

import torchlinops_gb300 as T
from torchlinops_gb300 import _ext, interp

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-5

CASES = [
    # grid, points, width, pad
    ((8, 9, 10), 700, 4.0, "circular"),  # regions of 12 cells wrap more than once
    ((24, 20, 28), 1, 4.0, "circular"),
    ((40, 33, 37), 20000, 4.0, "zero"),
    ((16, 24, 32), 9000, 3.0, "circular"),
    ((16, 16), 300, 4.0, "circular"),
    ((90, 62), 20000, 4.0, "zero"),
    ((48, 50), 9000, 6.0, "circular"),
    ((33, 61), 9000, 8.0, "zero"),
    ((64, 40), 9000, 5.5, "circular"),
    ((64, 40), 9000, 2.0, "circular"),
]


@pytest.mark.parametrize("shape,npts,width,pad", CASES)
@pytest.mark.parametrize("nb", [1, 2, 3, 5, 13])
def test_gather_against_oracle(shape, npts, width, pad, nb):
    gen = torch.Generator().manual_seed(npts + nb)
    n = torch.tensor(shape, dtype=torch.float32)
    locs = torch.rand(npts, len(shape), generator=gen) * (n + 4) - 2
    if npts > 1:
        locs[: npts // 2] = n / 3 + torch.rand(npts // 2, len(shape), generator=gen) * 6  # several items of a tile
        locs[:64] = torch.randint(-1, min(shape) + 1, (64, len(shape)), generator=gen).float()
        locs[64, 0] = float("nan")
    img = torch.complex(torch.randn(nb, *shape, generator=gen), torch.randn(nb, *shape, generator=gen))
    beta = OI.nufft_beta(width, 1.25)
    kw = dict(kernel="spline" if nb == 3 else "kaiser_bessel", pad_mode=pad)
    _ext.device_status(clear=True)
    got = T.ungrid(img.to(DEV), locs.to(DEV), width, kernel_params=dict(beta=beta), **kw).cpu()
    assert _ext.device_status() == 0
    want = OI.ungrid(img, torch.nan_to_num(locs), width, beta=beta, **kw)
    if npts > 1:
        assert bool((got[:, 64] == 0).all())  # a point without coordinates reads as zero
        got, want = got[:, torch.arange(npts) != 64], want[:, torch.arange(npts) != 64]
    assert rel_l2(got, want) < TOL


@pytest.mark.parametrize("nb", [4, 6])
def test_random_order_goes_through_the_items_order(nb):
    """Points in random order with a large output: the results are sorted back
    by a second pass, with the same sums as the direct stores."""
    import ctypes

    npts, size = (48 << 20) // (8 * nb) + 77, (40, 44, 48)
    gen = torch.Generator().manual_seed(nb)
    locs = torch.rand(npts, 3, generator=gen) * torch.tensor(size)
    locs[5] = float("inf")  # no taps: reads as zero
    img = torch.complex(torch.randn(nb, *size, generator=gen), torch.randn(nb, *size, generator=gen)).to(DEV)
    locs = locs.to(DEV)
    plan = interp.get_plan(locs, size, 4.0, "kaiser_bessel", "circular", 7.0)
    assert plan.scattered
    got = T.ungrid(img, locs, 4.0, kernel_params=dict(beta=7.0))
    d = interp._desc(3, size, (4.0,) * 3, "kaiser_bessel", 1, "circular", 7.0, True, nb, npts)
    sb = ctypes.c_size_t(0)
    assert _ext.lib().tlgb_interp_forward_scratch_size(ctypes.byref(d), ctypes.byref(plan.info), ctypes.byref(sb)) == 0
    assert sb.value == -(-nb // 4) * npts * 32
    direct = torch.empty_like(got)
    assert _ext.lib().tlgb_interp_forward(ctypes.byref(d), ctypes.byref(plan.info), _ext.ptr(plan.buffer), _ext.ptr(locs),
                                          _ext.ptr(img), _ext.ptr(direct), _ext.stream_ptr(locs.device)) == 0
    assert torch.equal(got, direct) and bool((got[:, 5] == 0).all())


def test_points_in_runs_are_stored_directly():
    locs = (20 + torch.arange(40000)[:, None] % 512 * 0.01 + torch.rand(1, 3)).to(DEV)
    assert not interp.get_plan(locs, (40, 40, 40), 4.0, "kaiser_bessel", "circular", 7.0).scattered
