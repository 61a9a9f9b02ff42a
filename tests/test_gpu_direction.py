"""Which direction the auto form takes, seen in the launches of the call after: classify, push and gate for a
push, the pull kernel alone for a pull.  Several warps count beside a hinted pull."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LINES = {"bin_bin_bin": {4: 18, 8: 27, 16: 45, 32: 41}, "bin_bin_count": {4: 18, 8: 14, 16: 12, 32: 8},
         "bin_bin_full": {4: 18, 8: 14, 16: 12, 32: 8}}


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("variant", list(LINES))
def test_direction_follows_the_share(pkg, cuda, T, variant):
    """A band matrix, where every tile-column holds as many tiles."""
    nbc = 5000
    n = nbc * T
    rows = np.repeat(np.arange(0, n, T), 3)
    cols = (rows + np.tile([0, 5 * T, 11 * T], nbc)) % n
    A = pkg.B2SRMatrix.from_graph(pkg.from_edges(rows, cols, nrows=n, ncols=n, drop_self_loops=False), T, device=cuda)
    assert A.nblocks == 3 * nbc
    A.set_launch(variant, direction="auto")
    fn, lib = getattr(A, "spmv_" + variant), pkg._lib.load()
    line = LINES[variant][T]
    perm = torch.randperm(nbc, generator=torch.Generator().manual_seed(T))
    for percent, push in ((line - 1, True), (line + 1, False), (100, False), (line - 1, True), (0, True),
                          (line, False), (1, True), (line + 1, False)):
        words = torch.zeros(nbc, dtype=torch.int64)
        words[perm[: nbc * percent // 100]] = 5
        x = words.to(pkg.word_dtype(T)).to(cuda)
        torch.cuda.synchronize()
        fn(x)  # follows the hint before; records its own share
        torch.cuda.synchronize()
        fn(x)
        assert lib.b2sr_last_launch_count() == (3 if push else 1), (percent, push)
    A.close()
