"""pad_shift and crop_shift of few entries or coils, which keep fewer of them in
flight: every entry of a batch as alone, bit for bit, and a crop's coils in order."""

import pytest
import torch

from torchlinops_gb300 import linops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im,padded", [((6, 5, 8), (7, 9, 10)), ((70, 64), (87, 80))])
@pytest.mark.parametrize("nb", [2, 3, 4, 5, 7, 9])
def test_entries_as_alone(im, padded, nb):
    gen = torch.Generator().manual_seed(nb)
    x = torch.randn(nb, *im, dtype=torch.complex64, generator=gen).cuda()
    z = torch.randn(nb, *padded, dtype=torch.complex64, generator=gen).cuda()
    apod = (torch.rand(*im, generator=gen) + 0.5).cuda()
    p, c = (linops.pad_shift(x, im, padded, apod=apod, modulate=True), linops.crop_shift(z, im, padded, apod=apod, modulate=True))
    for b in range(nb):
        assert torch.equal(p[b], linops.pad_shift(x[b:b + 1], im, padded, apod=apod, modulate=True)[0])
        assert torch.equal(c[b], linops.crop_shift(z[b:b + 1], im, padded, apod=apod, modulate=True)[0])


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 7, 9])
@pytest.mark.parametrize("nb", [1, 3])
def test_coils(C, nb):
    im, padded = (12, 10, 9), (15, 14, 9)
    gen = torch.Generator().manual_seed(C)
    maps = torch.randn(C, *im, dtype=torch.complex64, generator=gen).cuda()
    z = torch.randn(nb, C, *padded, dtype=torch.complex64, generator=gen).cuda()
    got = linops.crop_shift(z, im, padded, maps=maps, modulate=True)
    one = linops.crop_shift(z.reshape(nb * C, *padded), im, padded, modulate=True).reshape(nb, C, *im)
    want = (maps.to(torch.complex128).conj() * one).sum(1)
    torch.testing.assert_close(got, want.to(torch.complex64), rtol=2e-6, atol=2e-6 * C ** 0.5)  # C roundings of order-1 products
