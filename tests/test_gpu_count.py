"""Counts on full tiles, where every lane of a task adds its most: rows of 1 to 1300 tiles (each
bin of short rows, a whole task, several tasks), against the known degree and the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import from_np_words

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_counts_of_full_tiles(pkg, orc, cuda, T):
    ntiles = [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65, 128, 129, 255, 256, 257, 512, 513, 1300, 0, 1]
    nrows, ncols = len(ntiles) * T - 1, 1300 * T
    rows = np.concatenate([np.repeat(np.arange(i * T, min(i * T + T, nrows)), n * T) for i, n in enumerate(ntiles)])
    cols = np.concatenate([np.tile(np.arange(n * T), min(T, nrows - i * T)) for i, n in enumerate(ntiles)])
    g = pkg.from_edges(rows, cols, nrows=nrows, ncols=ncols, drop_self_loops=False)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    brp, bci, tiles = orc.csr_to_b2sr(g.rowptr, g.colind, g.nrows, T)
    rng = np.random.default_rng(T)
    for on in (np.ones(ncols, np.float32), (rng.random(ncols) < 0.5).astype(np.float32)):
        xb = orc.pack_vec_bits(on, T)
        xt = from_np_words(xb, T, cuda)
        want = orc.bmv_bin_bin_count(T, brp, bci, tiles, xb)
        if on.all():
            np.testing.assert_array_equal(want[:nrows], np.repeat(np.array(ntiles) * T, T)[:nrows])
        cnt = A.spmv_bin_bin_count(xt)
        np.testing.assert_array_equal(cnt.cpu().numpy(), want)
        full = A.spmv_bin_bin_full(xt)
        np.testing.assert_array_equal(full.cpu().numpy(), want.astype(np.float32))
        np.testing.assert_array_equal(A.spmv_bin_bin_count(xt, cnt.clone(), accumulate=True).cpu().numpy(), 2 * want)
        np.testing.assert_array_equal(A.spmv_bin_bin_full(xt, full.clone(), accumulate=True).cpu().numpy(),
                                      2 * want.astype(np.float32))
    A.close()


@pytest.mark.parametrize("T,percent", [(4, 18), (8, 14), (16, 12), (32, 8), (8, 27), (16, 45), (32, 41)])
def test_auto_direction_around_its_lines(pkg, cuda, T, percent):
    """A band matrix, where tile-columns hold equal numbers of tiles: frontiers of a share of the
    tile-columns just below, at and above each line, in turn, so that the next call's hint is wrong."""
    n = 200 * T
    rows = np.repeat(np.arange(n), 3)
    cols = (rows + np.tile([0, 5 * T, 11 * T], n)) % n
    A = pkg.B2SRMatrix.from_graph(pkg.from_edges(rows, cols, nrows=n, ncols=n, drop_self_loops=False), T, device=cuda)
    dt = pkg.word_dtype(T)
    for share in (percent - 1, percent, percent + 1, percent - 2, 100, 0, percent):
        words = torch.zeros(A.nblockcols, dtype=torch.int64)
        words[torch.randperm(200, generator=torch.Generator().manual_seed(share))[: 2 * share]] = 5
        xt = words.to(dt).to(cuda)
        got = {}
        for d in ("pull", "auto"):
            for v in ("bin_bin_bin", "bin_bin_count", "bin_bin_full"):
                A.set_launch(v, direction=d)
            got[d] = (A.spmv_bin_bin_bin(xt), A.spmv_bin_bin_count(xt), A.spmv_bin_bin_full(xt))
        for a, b in zip(got["auto"], got["pull"]):
            assert torch.equal(a, b), (share, T)
    A.close()
