"""Plans whose (point, block) pairs are counted before their memory is allocated:
the count, the same lists and the same grid as with room for the most pairs a point
can have, less memory, and a count that is too small refused with nothing written
past the buffers."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import binning as OB

import torchlinops_gb300 as T
from torchlinops_gb300 import _ext, interp

pytestmark = pytest.mark.gpu

CASES = [((25, 30, 27), 4.0, "circular"), ((24, 30, 29), 6.0, "zero"), ((33, 49), 4.0, "circular")]


def _locs(shape, npts, gen):
    n = torch.tensor(shape, dtype=torch.float32)
    locs = torch.rand(npts, len(shape), generator=gen) * (n + 4) - 2
    locs[: npts // 4] = n - 0.5 + torch.rand(npts // 4, len(shape), generator=gen)  # around the wrap
    locs[3] = float("nan")
    return locs


@pytest.mark.parametrize("shape,width,pad", CASES)
@pytest.mark.parametrize("npts", [1, 257, 6000])
def test_count_and_lists(shape, width, pad, npts, monkeypatch):
    gen = torch.Generator().manual_seed(npts)
    locs = _locs(shape, max(npts, 4), gen)[:npts]
    want = len(OB.block_pairs(locs, shape, width, "kaiser_bessel", pad, rows=3)[0])
    ld = locs.cuda()
    plain = interp.InterpolatePlan(ld, shape, width, "kaiser_bessel", pad, 7.0)
    monkeypatch.setattr(interp, "COUNT_POINTS", 0)
    counted = interp.InterpolatePlan(ld, shape, width, "kaiser_bessel", pad, 7.0)
    assert int(counted.info.n_blk_entries) == int(plain.info.n_blk_entries) == want
    assert counted.buffer.numel() < plain.buffer.numel() or npts < 300
    for off, count in (("off_blk_entries", want), ("off_blk_items", 4 * int(plain.info.n_blk_items)),
                       ("off_blk_split", 4 * int(plain.info.n_blk_split))):
        a, b = (p.buffer[int(getattr(p.info, off)):int(getattr(p.info, off)) + 4 * count] for p in (plain, counted))
        assert torch.equal(a, b)
    vals = torch.randn(3, npts, dtype=torch.complex64, generator=gen).cuda()
    kw = dict(pad_mode=pad, kernel_params=dict(beta=7.0))
    monkeypatch.undo()
    interp.clear_plan_cache()
    a = T.grid(vals, ld, shape, width, **kw)
    interp.clear_plan_cache()
    monkeypatch.setattr(interp, "COUNT_POINTS", 0)
    assert torch.equal(T.grid(vals, ld, shape, width, **kw), a)
    interp.clear_plan_cache()


def test_a_count_that_is_too_small_is_refused():
    shape, npts = (25, 30, 27), 5000
    ld = _locs(shape, npts, torch.Generator().manual_seed(1)).cuda()
    L = _ext.lib()
    d = interp._desc(3, shape, (4.0,) * 3, "kaiser_bessel", 1, "circular", 7.0, False, 1, npts)
    pb, tb = ctypes.c_size_t(0), ctypes.c_size_t(0)
    pairs = int(interp.InterpolatePlan(ld, shape, 4.0, "kaiser_bessel", "circular", 7.0).info.n_blk_entries)
    for count, ok in ((pairs, True), (pairs - 1, False), (pairs // 3, False), (0, False)):
        assert L.tlgb_interp_plan_size_counted(ctypes.byref(d), count, ctypes.byref(pb), ctypes.byref(tb)) == 0
        plan = torch.full((pb.value + 4096,), 77, dtype=torch.uint8, device="cuda")
        tmp = torch.full((tb.value + 4096,), 77, dtype=torch.uint8, device="cuda")
        info = _ext.PlanInfo()
        st = L.tlgb_interp_plan_build_counted(ctypes.byref(d), count, _ext.ptr(ld), _ext.ptr(plan), pb.value, _ext.ptr(tmp),
                                              tb.value, ctypes.byref(info), _ext.stream_ptr(ld.device))
        assert st == (_ext.TLGB_OK if ok else _ext.TLGB_ERR_INVALID)
        assert bool((plan[pb.value:] == 77).all()) and bool((tmp[tb.value:] == 77).all())


def test_memory_of_a_large_plan():
    """Evenly spread points of a circular 3D grid with cut last blocks: 144 bytes of
    rows, 64 of records, 32 of tile pairs, about 22 of block pairs and 4 per point."""
    shape, npts = (125, 150, 135), 600_000
    gen = torch.Generator().manual_seed(2)
    ld = (torch.rand(npts, 3, generator=gen) * torch.tensor(shape)).cuda()
    plan = interp.InterpolatePlan(ld, shape, 4.0, "kaiser_bessel", "circular", 7.0)
    assert int(plan.info.n_blk_items) > 0
    items = 16 * (2 * int(plan.info.n_tiles) + 3 * 35 * 40 * 40)
    assert plan.buffer.numel() < 285 * npts + items
    assert np.isfinite(plan.beta)
