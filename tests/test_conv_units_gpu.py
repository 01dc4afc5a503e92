"""Convolution layers at sizes that take work units of one, two, odd and many
rows, with a short last unit and with a last round that is not full, against the
float64 CPU oracle (float32 accumulation of exact products: 1e-5)."""

import pytest
import torch

from conftest import rel_l2
from oracle import conv as OC

from torchlinops_gb300 import _ext
from torchlinops_gb300 import precond as P

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("shape", [(24, 24, 24), (5, 7, 9), (128, 19, 33), (40, 50, 130), (100, 61, 12), (700, 3, 4)])
def test_conv_layer(shape):
    gen = torch.Generator().manual_seed(sum(shape))
    x = torch.randn(*shape, 16, generator=gen).to(torch.bfloat16)
    gy = torch.randn(*shape, 16, generator=gen).to(torch.bfloat16)
    w = (torch.randn(27, 16, 16, generator=gen) * 0.2).to(torch.bfloat16)
    _ext.device_status(clear=True)
    y = P.conv3d(x.to(DEV), w.to(DEV), out_f32=True).cpu()
    assert rel_l2(y.double(), OC.conv3d(x, w)) < 1e-5
    dw = P.conv3d_wgrad(x.to(DEV), gy.to(DEV))
    assert rel_l2(dw.cpu().double(), OC.conv3d_wgrad(x, gy)) < 1e-5
    assert torch.equal(dw, P.conv3d_wgrad(x.to(DEV), gy.to(DEV)))
    assert _ext.device_status() == 0
