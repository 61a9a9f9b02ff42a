"""Task lists built on the device (b2sr_plan.cu), through the multiplies that use them: tile-row counts
around a block of 1024, rows of every bin and at the segment lengths, long rows next to each other, and
wrapped arrays whose rowptr is not monotone (refused)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(pkg, T, tile_rows, seed):
    """Tile-rows whose tile counts run over the bins and the segment lengths, in a shuffled order."""
    rng = np.random.default_rng(seed)
    sizes = [0, 1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 512, 513, 1100, 2500]
    m = np.array([sizes[i % len(sizes)] if i < 60 else rng.integers(0, 12) for i in range(tile_rows)])
    rng.shuffle(m)
    m[: min(40, tile_rows)] = 700  # long rows side by side
    nbc = 3000
    rows = np.concatenate([np.full(c, i * T + int(rng.integers(0, T))) for i, c in enumerate(m)] + [np.zeros(0, int)])
    cols = np.concatenate([rng.choice(nbc, c, replace=False) * T for c in m] + [np.zeros(0, int)])
    cols = cols + rng.integers(0, T, cols.size)
    return pkg.from_edges(rows, cols, nrows=tile_rows * T, ncols=nbc * T, drop_self_loops=False)


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("tile_rows", [1, 31, 1023, 1024, 1025, 5000])
def test_every_row_once(pkg, cuda, T, tile_rows):
    g = _graph(pkg, T, tile_rows, T + tile_rows)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    deg = g.degrees()
    ones = torch.ones(g.ncols, device=cuda)
    np.testing.assert_array_equal(A.spmv_bin_full_full(ones).cpu().numpy()[: g.nrows], deg.astype(np.float32))
    bits = A.pack_bits(ones)
    np.testing.assert_array_equal(A.spmv_bin_bin_count(bits).cpu().numpy()[: g.nrows], deg)
    for k in (3, 64):
        X = torch.arange(1, k + 1, device=cuda, dtype=torch.float32).expand(g.ncols, k).contiguous()
        want = deg[:, None].astype(np.float32) * np.arange(1, k + 1, dtype=np.float32)
        np.testing.assert_array_equal(A.spmm(X).cpu().numpy()[: g.nrows], want)
    A.close()


def test_rowptr_that_asks_for_more_than_its_tiles(pkg, cuda):
    """A wrapped rowptr that runs past the tiles and back: no plan, no launch."""
    nb, nt = 2000, 64
    rp = np.zeros(nb + 1, np.int32)
    rp[1::2] = 1 << 20  # every other tile-row claims a million tiles
    rp[-1] = nt
    A = pkg.B2SRMatrix.wrap(torch.from_numpy(rp).to(cuda), torch.zeros(nt, dtype=torch.int32, device=cuda),
                            torch.zeros(nt * 8, dtype=torch.uint8, device=cuda), nb * 8, 80, 8)
    with pytest.raises(pkg.B2SRError) as e:
        A.spmv_bin_full_full(torch.ones(80, device=cuda))
    assert e.value.status in (1, 6)
    A.close()
