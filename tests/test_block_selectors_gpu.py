"""The block lists' entries in full (point and block selector) and the blocks of
their work items against the CPU oracle, for two and three rows per dimension."""

import numpy as np
import pytest
import torch

from oracle import binning as OB

from torchlinops_gb300 import interp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,width,pad,rows", [((25, 30, 27), 4.0, "circular", 3), ((8, 9, 11), 4.0, "circular", 3),
                                                  ((24, 30, 29), 6.0, "zero", 3), ((20, 33, 26), 8.0, "zero", 3),
                                                  ((33, 49), 4.0, "circular", 3), ((48, 50), 6.0, "circular", 3),
                                                  ((24, 28, 32), 4.0, "circular", 2), ((40, 61), 6.0, "zero", 2)])
def test_entries_and_items(shape, width, pad, rows):
    gen = torch.Generator().manual_seed(sum(shape))
    n = torch.tensor(shape, dtype=torch.float32)
    locs = torch.cat([torch.rand(5000, len(shape), generator=gen) * (n + 6) - 3,
                      n - 0.5 + torch.rand(2000, len(shape), generator=gen),  # around the wrap, split blocks
                      torch.randint(-2, min(shape) + 2, (200, len(shape)), generator=gen).float()])
    locs[:7, 0] = float("nan")
    keys, entries = OB.block_pairs(locs, shape, width, "kaiser_bessel", pad, rows=rows)
    plan = interp.InterpolatePlan(locs.cuda(), shape, width, "kaiser_bessel", pad, 7.0)
    info = plan.info

    def words(off, count):
        return plan.buffer[int(off):int(off) + 4 * int(count)].view(torch.int32).cpu().numpy()

    got = words(info.off_blk_entries, info.n_blk_entries).astype(np.int64) & 0xFFFFFFFF
    assert np.array_equal(got, entries)
    items = words(info.off_blk_items, 4 * int(info.n_blk_items)).reshape(-1, 4)
    seen = np.zeros(len(entries), dtype=int)
    for b, q0, q1, _ in items[items[:, 1] < items[:, 2]]:
        assert np.all(keys[q0:q1] == b)
        seen[q0:q1] += 1
    assert np.all(seen == 1)
