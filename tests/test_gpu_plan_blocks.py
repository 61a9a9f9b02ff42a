"""Task lists (b2sr_plan.cu) of tile-row counts around the 256 of a block, with cut tile-rows at the
edges of the blocks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("tile_rows", [255, 256, 257, 511, 512, 513, 769])
def test_every_row_once(pkg, cuda, T, tile_rows):
    rng = np.random.default_rng(T + tile_rows)
    m = rng.integers(0, 10, tile_rows)
    for at in (0, 31, 32, 254, 255, 256, 257, 511, 512, tile_rows - 1):
        if at < tile_rows:
            m[at] = rng.integers(600, 1400)
    rows = np.concatenate([np.full(c, i * T + int(rng.integers(0, T))) for i, c in enumerate(m)])
    cols = np.concatenate([rng.choice(1500, c, replace=False) * T for c in m]) + rng.integers(0, T, rows.size)
    g = pkg.from_edges(rows, cols, nrows=tile_rows * T, ncols=1500 * T, drop_self_loops=False)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    deg, ones = g.degrees(), torch.ones(g.ncols, device=cuda)
    np.testing.assert_array_equal(A.spmv_bin_full_full(ones).cpu().numpy(), deg.astype(np.float32))
    np.testing.assert_array_equal(A.spmv_bin_bin_count(A.pack_bits(ones)).cpu().numpy(), deg)
    np.testing.assert_array_equal(A.spmm(ones[:, None].repeat(1, 5)).cpu().numpy()[:, 4], deg.astype(np.float32))
    A.close()
