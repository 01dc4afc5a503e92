"""Consumers that give up while copies into their CTA's shared memory are under way:
the producers still end with every copy landed, the failure is reported, and the
passes that follow are right. The hook's waits for copies give up at once; a CTA
has one unit at most, so its producers never wait for a consumer that has left."""

import pytest
import torch

from conftest import rel_l2
from oracle import interp as OI

import torchlinops_gb300 as T
from torchlinops_gb300 import _ext, interp

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture
def hook():
    L = _ext.lib()
    yield L
    L.tlgb_test_skip_region_copy(0)
    _ext.device_status(clear=True)


# by TMA, and by plain copies (odd last extent)
@pytest.mark.parametrize("shape", [(32, 24, 32), (24, 24, 31), (48, 64), (48, 61)])
def test_gather_and_gradient(hook, shape):
    gen = torch.Generator().manual_seed(sum(shape))
    npts, kp = 500, dict(beta=T.kaiser_bessel_beta(4.0, 1.25))
    locs = torch.rand(npts, len(shape), generator=gen) * torch.tensor(shape)
    img = torch.randn(4, *shape, dtype=torch.complex64, generator=gen)
    a = torch.randn(4, npts, dtype=torch.complex64, generator=gen).to(DEV)
    locs_d, img_d = locs.to(DEV), img.to(DEV)
    plan = interp.get_plan(locs_d, shape, 4.0, "kaiser_bessel", "circular", kp["beta"])
    assert plan.info.n_fwd_items <= torch.cuda.get_device_properties(0).multi_processor_count  # units <= CTAs
    want = OI.ungrid(img, locs, 4.0, beta=kp["beta"])
    grad = interp._grad_locs(img_d, a, locs_d, 4.0, "kaiser_bessel", 1, "circular", kp)
    _ext.device_status(clear=True)
    for _ in range(20):
        hook.tlgb_test_skip_region_copy(2)
        T.ungrid(img_d, locs_d, 4.0, kernel_params=kp)
        if len(shape) == 2:
            interp._grad_locs(img_d, a, locs_d, 4.0, "kaiser_bessel", 1, "circular", kp)
        assert hook.tlgb_test_skip_region_copy(0) == 2
        got = T.ungrid(img_d, locs_d, 4.0, kernel_params=kp)  # right behind the failed passes
        assert rel_l2(got.cpu(), want) < 1e-5
        assert torch.equal(interp._grad_locs(img_d, a, locs_d, 4.0, "kaiser_bessel", 1, "circular", kp), grad)
        assert _ext.device_status(clear=True) & 1
    T.ungrid(img_d, locs_d, 4.0, kernel_params=kp)
    assert _ext.device_status() == 0
