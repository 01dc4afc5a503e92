"""The interpolation calls take norm 1 or 2 as an int and refuse everything else,
also where a plan of the same points is already there."""

import pytest
import torch

import torchlinops_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm,error", [(1.5, ValueError), (0, ValueError), (3, ValueError), ("1", ValueError),
                                        (1.0, TypeError), (2.0, TypeError)])
def test_refused(norm, error):
    img, locs = torch.randn(1, 16, 16, device="cuda"), torch.rand(9, 2, device="cuda") * 16
    T.ungrid(img, locs, 4.0, norm=1)
    pts = T.ungrid(img, locs, 4.0, norm=2)
    for f in (T.ungrid, T.interpolate):
        with pytest.raises(error):
            f(img, locs, 4.0, norm=norm)
    for f in (T.grid, T.interpolate_adjoint):
        with pytest.raises(error):
            f(pts, locs, (16, 16), 4.0, norm=norm)
