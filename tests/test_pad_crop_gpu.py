"""pad_shift and crop_shift over batches around the groups of 8 entries that a
thread keeps in flight and over runs of several groups, with and without coil
maps, against torch; and the functional NUFFT, whose scales are in the
apodization weights."""

import pytest
import torch

from torchlinops_gb300 import linops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("im,padded", [((6, 5, 8), (7, 9, 10)), ((12, 9), (15, 9)), ((70, 64), (87, 80)), ((5,), (1201,))])
@pytest.mark.parametrize("nb,C", [(1, 0), (7, 0), (8, 0), (17, 0), (300, 0), (1, 1), (1, 9), (3, 8), (5, 11), (40, 2)])
@pytest.mark.parametrize("modulate", [False, True])
def test_batches_against_torch(im, padded, nb, C, modulate):
    gen = torch.Generator().manual_seed(nb + C)
    nd = len(im)
    dims = tuple(range(-nd, 0))
    x = torch.randn(nb, *im, dtype=torch.complex64, generator=gen)
    maps = torch.randn(C, *im, dtype=torch.complex64, generator=gen) if C else None
    apod = torch.rand(*im, generator=gen) + 0.5
    pad = linops.pad_to_size(im, padded)
    m = torch.ones(padded, dtype=torch.complex128)
    if modulate:
        for e, p in enumerate(padded):
            ph = torch.exp(2j * torch.pi * ((torch.arange(p, dtype=torch.float64) * (p // 2)) % p) / p)
            m = m * ph.reshape([-1 if d == e else 1 for d in range(nd)])
    src = apod * x if maps is None else maps * (apod * x)[:, None]
    ref = torch.fft.ifftshift(torch.nn.functional.pad(src, pad), dim=dims) * m
    mg = None if maps is None else maps.to(DEV)
    got = linops.pad_shift(x.to(DEV), im, padded, maps=mg, apod=apod.to(DEV), modulate=modulate).cpu()
    torch.testing.assert_close(got, ref.to(torch.complex64), rtol=2e-6, atol=2e-6)
    z = torch.randn(*src.shape[:-nd], *padded, dtype=torch.complex64, generator=gen)
    sl = (Ellipsis,) + tuple(linops.crop_slice_from_pad(pad))
    back = torch.fft.fftshift(z * m.conj(), dim=dims)[sl]
    if maps is not None:
        back = (maps.conj() * back).sum(1)
    add = torch.randn(nb, *im, dtype=torch.complex64, generator=gen)
    gotb = linops.crop_shift(z.to(DEV), im, padded, maps=mg, apod=apod.to(DEV), alpha=0.5, add=add.to(DEV), beta=2.0,
                             modulate=modulate).cpu()
    torch.testing.assert_close(gotb, (0.5 * apod * back + 2.0 * add).to(torch.complex64), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("grid_size", [(20, 17), (10, 12, 9)])
def test_functional_nufft_has_the_scale_of_the_operator(grid_size):
    """The functional transforms against the operator that scales after its FFT."""
    gen = torch.Generator().manual_seed(2)
    locs = ((torch.rand(300, len(grid_size), generator=gen) - 0.5) * torch.tensor(grid_size)).to(DEV)
    x = torch.randn(3, *grid_size, dtype=torch.complex64, generator=gen).to(DEV)
    A = linops.NUFFT(locs, grid_size)
    y = linops.nufft(x, locs)
    torch.testing.assert_close(y, A(x), rtol=1e-5, atol=1e-5 * float(y.abs().max()))
    b = linops.nufft_adjoint(y, locs, grid_size)
    torch.testing.assert_close(b, A.H(y), rtol=1e-5, atol=1e-5 * float(b.abs().max()))
