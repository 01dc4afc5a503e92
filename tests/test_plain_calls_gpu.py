"""Calls that skip the autograd Function when no input requires a gradient:
whatever watches a call (forward-mode AD, functorch, tracing, another stream)
still sees what it saw, and layouts that need a copy still get one."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD

import torchlinops_gb300 as T
from torchlinops_gb300 import _ext

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def case():
    gen = torch.Generator().manual_seed(8)
    img = torch.randn(3, 20, 24, dtype=torch.complex64, generator=gen).to(DEV)
    locs = (torch.rand(500, 2, generator=gen) * 20).to(DEV)
    return img, locs


def _ops(img, locs):
    idx = (locs[:, 0].long(), locs[:, 1].long())
    pts = T.interpolate(img, locs, 4.0)
    return [
        (img, lambda v: T.interpolate(v, locs, 4.0)),
        (pts, lambda v: T.interpolate_adjoint(v, locs, (20, 24), 4.0)),
        (img, lambda v: T.index(v, idx)),
        (pts, lambda v: T.index_adjoint(v, idx, (20, 24))),
        (img, lambda v: T.array_to_blocks(v, (4, 4), (2, 2))),
    ]


def test_forward_mode_is_refused_not_dropped(case):
    for x, f in _ops(*case):
        with fwAD.dual_level():
            with pytest.raises((NotImplementedError, RuntimeError)):
                f(fwAD.make_dual(x, torch.ones_like(x)))


def test_functorch_gradients_are_right_or_refused(case):
    """The interpolation's backward refuses wrapped tensors; no operator may
    return a gradient of zero for a call that skipped its Function."""
    for x, f in _ops(*case):
        r = x.real.contiguous().requires_grad_(True)
        want = torch.autograd.grad((f(r) ** 2).sum(), r)[0]
        try:
            got = torch.func.grad(lambda v: (f(v) ** 2).sum())(r.detach())
        except RuntimeError:
            continue
        assert torch.equal(got, want)


def test_same_results_with_and_without_a_gradient(case):
    for x, f in _ops(*case):
        y = f(x.clone().requires_grad_(True))
        assert y.requires_grad and not f(x).requires_grad
        assert torch.equal(f(x), y.detach())
        with torch.no_grad():
            assert torch.equal(f(x.clone().requires_grad_(True)), y.detach())


def test_layouts_that_need_a_copy(case):
    img, locs = case
    want = T.interpolate(img, locs, 4.0)
    assert torch.equal(T.interpolate(img.transpose(1, 2).contiguous().transpose(1, 2), locs, 4.0), want)
    assert torch.equal(T.interpolate(img.conj().resolve_conj().conj(), locs, 4.0), want)
    assert torch.equal(T.interpolate(img, locs.double(), 4.0), want)
    assert torch.equal(T.interpolate(img, locs.T.contiguous().T, 4.0), want)
    assert torch.equal(T.interpolate(img[:0], locs, 4.0), want[:0])


def test_other_streams_see_the_plan(case):
    img, locs = case
    want = T.interpolate(img, locs, 4.0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert _ext.raw_stream(img.device) == side.cuda_stream
        got = T.interpolate(img, locs, 4.0)
        built_there = T.interpolate(img, locs.clone(), 4.0)
    side.synchronize()
    assert torch.equal(got, want) and torch.equal(built_there, want)
