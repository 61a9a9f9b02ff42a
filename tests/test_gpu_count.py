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
