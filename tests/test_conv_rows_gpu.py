"""Convolution layers with more rows than one work unit and more units than
CTAs: row segments of 16 and their remainders, the rings' wrap-around, ragged
column tiles, against the float64 CPU oracle (float32 accumulation of exact
products: 1e-5)."""

import pytest
import torch

from conftest import rel_l2
from oracle import conv as OC

from torchlinops_gb300 import _ext
from torchlinops_gb300 import precond as P

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("shape", [(2, 16, 129), (3, 37, 140), (150, 33, 20), (1, 200, 64), (333, 1, 5)])
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
