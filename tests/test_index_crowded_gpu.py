"""Sampling adjoint with samples crowded into few cells of a mostly empty grid, and
on both sides of the densities at which its kernels change, for every element
size: bit for bit the sequential sum over the samples."""

import pytest
import torch

from oracle import index as OX

import torchlinops_gb300 as T

pytestmark = pytest.mark.gpu

SHAPE = (30, 37, 41)  # 45510 cells: 45 and 178 runs of 1024 and 256, the last one cut
CELLS = 30 * 37 * 41


def _values(nb, n, dtype, gen):
    if dtype in (torch.int32, torch.int64):
        return torch.randint(-1000, 1000, (nb, n), generator=gen, dtype=dtype)
    return torch.randn(nb, n, generator=gen, dtype=dtype)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128, torch.float32, torch.int64])
@pytest.mark.parametrize("npts", [CELLS // 4 - 1, CELLS // 4 + 1, CELLS + 1, 2 * CELLS + 1])
@pytest.mark.parametrize("nb", [1, 2, 5])
@pytest.mark.parametrize("crowd", [False, True])
def test_adjoint_bit_for_bit(dtype, npts, nb, crowd):
    gen = torch.Generator().manual_seed(npts + nb)
    idx = [torch.randint(0, s, (npts,), generator=gen) for s in SHAPE]
    if crowd:  # three quarters of the samples in 12 neighbouring cells, the rest anywhere
        for i, (first, n) in zip(idx, ((7, 2), (36, 1), (30, 6))):
            i[npts // 4:] = first + torch.randint(0, n, (npts - npts // 4,), generator=gen)
    v = _values(nb, npts, dtype, gen)
    got = T.index_adjoint(v.cuda(), tuple(i.cuda() for i in idx), SHAPE)
    assert torch.equal(got.cpu(), OX.index_adjoint(v, tuple(idx), SHAPE))


@pytest.mark.parametrize("nb", [1, 3])
def test_many_samples_per_cell_of_16_bytes(nb):
    gen = torch.Generator().manual_seed(nb)
    idx = tuple(torch.randint(0, s, (40000,), generator=gen) for s in (31, 33))
    v = torch.randn(nb, 40000, generator=gen, dtype=torch.complex128)
    got = T.index_adjoint(v.cuda(), tuple(i.cuda() for i in idx), (31, 33))
    assert torch.equal(got.cpu(), OX.index_adjoint(v, idx, (31, 33)))
