"""T = 4 stores a row or an x word in the low half of a byte.  Wrapped tiles and x words whose upper halves
are not zero (a complement taken on bytes, a file of another writer) give the products of the lower halves,
in every form: short rows, whole tasks, rows cut into tasks; pull, push and the merge path."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dirt_a,dirt_x", [(0xF0, 0xF0), (0x50, 0xF0), (0x90, 0x10), (0xF0, 0)])
def test_unused_halves_do_not_count(pkg, orc, cuda, dirt_a, dirt_x):
    T = 4
    ntiles = [0, 1, 2, 3, 4, 5, 8, 9, 31, 64, 65, 128, 255, 256, 257, 600]
    rng = np.random.default_rng(dirt_a + dirt_x)
    rows = np.concatenate([i * T + rng.integers(0, T, 2 * n) for i, n in enumerate(ntiles)])
    cols = np.concatenate([rng.permutation(np.tile(np.arange(n) * T, 2)) + rng.integers(0, T, 2 * n) for n in ntiles])
    n, ncols = len(ntiles) * T, 600 * T
    g = pkg.from_edges(rows, cols, nrows=n, ncols=ncols, drop_self_loops=False)
    brp, bci, tiles = orc.csr_to_b2sr(g.rowptr, g.colind, n, T)
    xb = orc.pack_vec_bits((rng.random(ncols) < 0.4).astype(np.float32), T)
    mask = rng.integers(0, 256, len(brp) - 1).astype(np.uint8)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)  # noqa: E731
    A = pkg.B2SRMatrix.wrap(dev(brp), dev(bci), dev(tiles | np.uint8(dirt_a)), n, ncols, T)
    x, m = dev(xb | np.uint8(dirt_x)), dev(mask)
    bits = orc.bmv_bin_bin_bin(T, brp, bci, tiles, xb)
    cnt = orc.bmv_bin_bin_count(T, brp, bci, tiles, xb)
    for opt in ({}, {"direction": "push"}, {"direction": "auto"}, {"algorithm": "merge"}):
        for v in ("bin_bin_bin", "bin_bin_count", "bin_bin_full"):
            A.set_launch(v, **opt)
        for _ in range(2):  # auto: the second call follows the first one's hint
            np.testing.assert_array_equal(A.spmv_bin_bin_bin(x).cpu().numpy(), bits, err_msg=str(opt))
            np.testing.assert_array_equal(A.spmv_bin_bin_bin_masked(x, m).cpu().numpy(), bits & ~mask, err_msg=str(opt))
            np.testing.assert_array_equal(A.spmv_bin_bin_count(x).cpu().numpy(), cnt, err_msg=str(opt))
            np.testing.assert_array_equal(A.spmv_bin_bin_full(x).cpu().numpy(), cnt.astype(np.float32), err_msg=str(opt))
    A.close()
