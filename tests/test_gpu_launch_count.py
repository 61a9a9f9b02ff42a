"""b2sr_last_launch_count of a transpose: tile-rows, (count, scan, scatter) per digit pass, the row pointer,
and at T = 16 and 32 the gather; the scan of n counts is one launch up to 4096 of them, two up to 4096 * 1024."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("nbc,entries,passes,scan", [(1, 50, 1, 1), (500, 3000, 1, 1), (500, 60000, 1, 2), (5000, 3000, 2, 1)])
def test_transpose(pkg, cuda, T, nbc, entries, passes, scan):
    # one entry a tile: every (tile-row, tile-column) pair once
    pairs = np.arange(entries)
    g = pkg.from_edges(pairs // nbc * T, pairs % nbc * T, nrows=(entries // nbc + 1) * T, ncols=nbc * T, drop_self_loops=False)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    assert A.nblocks == entries
    digits = 1 << -(-max((nbc - 1).bit_length(), 1) // passes)
    assert (digits * -(-entries // 4096) > 4096) == (scan == 2)
    A.transpose()
    assert pkg._lib.load().b2sr_last_launch_count() == 2 + passes * (2 + scan) + (T >= 16)
    A.close()
