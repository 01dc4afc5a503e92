"""A NaN or Inf in one image cell reaches exactly the points whose window holds
the cell: kernels narrower than the gather's box of cells, windows cut by a zero-
padded edge, every group size, and the other points' results as on a finite image."""

import pytest
import torch

from conftest import rel_l2
from oracle import interp as OI

import torchlinops_gb300 as T
from torchlinops_gb300 import interp

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-5

SHAPES_2D = [(40, 33), (16, 48)]
SHAPES_3D = [(24, 17, 20), (16, 24, 32)]


def _case(shape, width, pad, nb, cell):
    gen = torch.Generator().manual_seed(int(10 * width) + nb + sum(shape))
    n = torch.tensor(shape, dtype=torch.float32)
    npts = 1500
    locs = torch.rand(npts, len(shape), generator=gen) * (n + 2) - 1
    at = torch.tensor(cell, dtype=torch.float32)
    locs[:900] = at + torch.rand(900, len(shape), generator=gen) * 2 * (width + 2) - (width + 2)  # windows around the cell
    locs[900:1000] = at + torch.randint(-5, 6, (100, len(shape)), generator=gen)  # exact-integer coordinates
    img = torch.complex(torch.randn(nb, *shape, generator=gen), torch.randn(nb, *shape, generator=gen))
    beta = OI.nufft_beta(width, 1.25)
    one = torch.zeros(1, *shape, dtype=torch.complex64)
    one[(0, *cell)] = 1.0
    hit = OI.ungrid(one, locs, width, beta=beta, pad_mode=pad)[0].abs() > 0  # a Kaiser-Bessel weight is never 0
    assert 0 < int(hit.sum()) < npts
    return locs, img, dict(beta=beta), hit


def _cells(shape):
    return [tuple(s // 2 for s in shape), tuple(0 if i else s - 1 for i, s in enumerate(shape))]


@pytest.mark.parametrize("shape,width", [(s, w) for s in SHAPES_2D for w in (2.0, 3.0, 3.5, 4.0, 5.5, 6.0, 8.0)]
                         + [(s, w) for s in SHAPES_3D for w in (2.0, 3.0, 3.5, 4.0)])
@pytest.mark.parametrize("pad", ["circular", "zero"])
@pytest.mark.parametrize("nb", [1, 2, 3, 9])
def test_ungrid(shape, width, pad, nb):
    for cell, value in zip(_cells(shape), (complex(float("nan"), 1.0), complex(2.0, float("-inf")))):
        locs, img, kp, hit = _case(shape, width, pad, nb, cell)
        good = T.ungrid(img.to(DEV), locs.to(DEV), width, pad_mode=pad, kernel_params=kp).cpu()
        img[(nb - 1, *cell)] = value
        got = T.ungrid(img.to(DEV), locs.to(DEV), width, pad_mode=pad, kernel_params=kp).cpu()
        assert torch.equal(got[:-1], good[:-1])  # the other entries of the points are the same bits
        finite = torch.isfinite(torch.view_as_real(got[-1])).all(-1)
        assert torch.equal(finite, ~hit)
        assert rel_l2(got[-1][~hit], good[-1][~hit]) < TOL


@pytest.mark.parametrize("shape", SHAPES_2D)
@pytest.mark.parametrize("width", [2.0, 3.0, 3.5, 4.0])
@pytest.mark.parametrize("pad", ["circular", "zero"])
@pytest.mark.parametrize("nb", [1, 3, 9, 40])
def test_trajectory_gradient(shape, width, pad, nb):
    for cell, value in zip(_cells(shape), (complex(float("nan"), 1.0), complex(2.0, float("-inf")))):
        locs, img, kp, hit = _case(shape, width, pad, nb, cell)
        gen = torch.Generator().manual_seed(nb)
        a = torch.complex(torch.randn(nb, len(locs), generator=gen), torch.randn(nb, len(locs), generator=gen)).to(DEV)
        img[(nb - 1, *cell)] = 0
        args = (a, locs.to(DEV), width, "kaiser_bessel", 1, pad, kp)
        good = interp._grad_locs(img.to(DEV), *args).cpu()
        img[(nb - 1, *cell)] = value
        got = interp._grad_locs(img.to(DEV), *args).cpu()
        finite = torch.isfinite(got).all(-1)
        assert torch.equal(finite, ~hit)
        assert torch.equal(got[~hit], good[~hit])  # the same sums without the cell
