"""Sampling and its adjoint over batches around the groups of entries and
samples that a thread keeps in flight, on grids that fill the device and on
small ones with many samples per cell, against torch on the CPU (bit for bit:
the adjoint adds in the order of a sequential index_add_)."""

import pytest
import torch

import torchlinops_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,npts", [((3, 4), 5000), ((1,), 77), ((130, 90), 2047), ((70, 80, 60), 2049), ((96, 96, 96), 70000), ((37, 41), 0)])
@pytest.mark.parametrize("nb", [1, 2, 3, 5, 8, 9, 21])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.float32, torch.int64])
def test_against_torch(size, npts, nb, dtype):
    gen = torch.Generator().manual_seed(npts + nb)
    idx = tuple(torch.randint(0, s, (npts,), generator=gen) for s in size)
    n = torch.tensor(size).prod().item()
    draw = (lambda *s: torch.randint(-99, 99, s, generator=gen)) if dtype == torch.int64 else (
        lambda *s: torch.randn(*s, generator=gen, dtype=dtype))
    img, vals = draw(nb, *size), draw(nb, npts)
    flat = torch.zeros(npts, dtype=torch.int64)
    for i, s in zip(idx, size):
        flat = flat * s + i
    didx = tuple(i.cuda() for i in idx)
    assert torch.equal(T.index(img.cuda(), didx).cpu(), img.reshape(nb, n)[:, flat])
    want = torch.zeros(nb, n, dtype=dtype)
    for b in range(nb):  # one entry at a time: a sequential sum in sample order
        want[b].index_add_(0, flat, vals[b])
    assert torch.equal(T.index_adjoint(vals.cuda(), didx, size).cpu().reshape(nb, n), want)


@pytest.mark.parametrize("dtype", [torch.bool, torch.float16, torch.complex128])
def test_element_sizes(dtype):
    gen = torch.Generator().manual_seed(1)
    img = torch.randn(40, 33, 50, generator=gen, dtype=torch.float64).to(dtype)
    idx = tuple(torch.randint(0, s, (5000,), generator=gen) for s in (33, 50))
    assert torch.equal(T.index(img.cuda(), tuple(i.cuda() for i in idx)).cpu(), img[:, idx[0], idx[1]])
