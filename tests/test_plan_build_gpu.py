"""The device-built plan at the edges of its kernels' tiles, against the CPU
oracle: no points, one point, a CTA of points and one more, a sort tile of
pairs and its remainders, and a grid with enough tiles for an odd number of
sort passes. The item lists cover every pair once."""

import numpy as np
import pytest
import torch

from oracle import binning as OB

from torchlinops_gb300 import interp

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [
    ((24, 20, 28), 1, "circular"),
    ((24, 20, 28), 256, "zero"),
    ((24, 20, 28), 257, "circular"),
    ((40, 36, 48), 4096, "circular"),
    ((64, 48), 4097, "circular"),
    ((700,), 4095, "circular"),
    ((7, 12, 13), 3000, "circular"),  # tile lists only: a window could meet a block twice
    ((520, 520, 520), 3000, "zero"),  # three sort passes
]


def _list(plan, off, n, width=1):
    raw = plan.buffer[int(off):int(off) + 4 * width * int(n)].view(torch.int32).cpu().numpy()
    return raw.reshape(-1, width) if width > 1 else raw


@pytest.mark.parametrize("grid_size,npts,pad", CASES)
def test_plan_lists_at_the_edges(grid_size, npts, pad):
    gen = torch.Generator().manual_seed(3 * npts + len(grid_size))
    n = torch.tensor(grid_size, dtype=torch.float32)
    locs = torch.rand(npts, len(grid_size), generator=gen) * (n + 4) - 2
    locs[: npts // 3] = n / 2 + torch.randn(npts // 3, len(grid_size), generator=gen)  # a dense centre
    keys, pts = OB.plan_pairs(locs, grid_size, 4.0, "kaiser_bessel", pad)
    plan = interp.InterpolatePlan(locs.to(DEV), grid_size, 4.0, "kaiser_bessel", pad, 6.99666)
    info = plan.info
    assert np.array_equal(_list(plan, info.off_entries, info.n_entries), pts)
    fwd = _list(plan, info.off_fwd_items, info.n_fwd_items, 4)
    seen = np.zeros(len(pts), dtype=int)
    for t, b, e, _ in fwd:  # home pairs, at most 512 to an item
        assert 0 < e - b <= 512 and np.all(keys[b:e] == 2 * t)
        seen[b:e] += 1
    assert np.array_equal(seen, (keys % 2 == 0).astype(int))
    adj = _list(plan, info.off_adj_items, info.n_adj_items, 4)
    seen[:] = 0
    for t, b, e, _ in adj:
        assert e - b <= int(info.chunk) and np.all(keys[b:e] // 2 == t)
        seen[b:e] += 1
    assert np.all(seen == 1)
    assert set(adj[:, 0]) == set(range(int(info.n_tiles)))  # empty tiles are written too
    assert np.all(np.diff(adj[:, 2] - adj[:, 1]) <= 0)
    if int(info.n_blk_items) > 0:
        bkeys, bpts = OB.block_pairs(locs, grid_size, 4.0, "kaiser_bessel", pad)
        got = _list(plan, info.off_blk_entries, info.n_blk_entries).astype(np.int64) & 0xFFFFFFFF
        assert np.array_equal(got, bpts)
        items = _list(plan, info.off_blk_items, info.n_blk_items, 4)
        full = items[items[:, 1] < items[:, 2]]
        seen = np.zeros(len(bpts), dtype=int)
        for b, s0, s1, _ in full:
            assert np.all(bkeys[s0:s1] == b)
            seen[s0:s1] += 1
        assert np.all(seen == 1)
        empty = items[items[:, 1] == items[:, 2]]
        nblk = int(np.prod([-(-s // (4 if len(grid_size) == 3 else 8)) for s in grid_size]))
        assert -empty[:, 3].sum() + len(np.unique(full[:, 0])) == nblk


def test_plan_without_points():
    plan = interp.InterpolatePlan(torch.zeros(0, 3, device=DEV), (24, 20, 28), 4.0, "kaiser_bessel", "circular", 1.0)
    assert int(plan.info.n_entries) == 0 and int(plan.info.n_fwd_items) == 0
    assert int(plan.info.n_adj_items) == int(plan.info.n_tiles)
