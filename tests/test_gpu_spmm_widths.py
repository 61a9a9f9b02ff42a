"""Dense-RHS widths on both sides of every lane layout of spmm_rows_kernel (b2sr_spmm_rows.cu), with
aligned and unaligned rows, against FP64 sums over the CSR."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import REL_TOL

pytestmark = pytest.mark.gpu

WIDTHS = [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 50, 63, 64, 65, 96, 97, 98, 128, 129, 160, 257]


@pytest.fixture(scope="module")
def graph(pkg):
    """Hubs (segments, full item lists), short and empty rows, and more columns than rows."""
    rng = np.random.default_rng(8)
    n, nc = 1003, 1300
    rows = np.concatenate([rng.integers(0, n, 6000), np.repeat([5, 6, 700], 1200), np.repeat(np.arange(64, 96), 400)])
    cols = np.concatenate([rng.integers(0, nc, 6000), np.tile(np.arange(1200), 3), np.tile(np.arange(300, 700), 32)])
    return pkg.from_edges(rows, cols, nrows=n, ncols=nc, drop_self_loops=False)


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_widths(pkg, cuda, graph, T, dtype):
    g = graph
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    row = torch.from_numpy(np.repeat(np.arange(g.nrows), np.diff(g.rowptr))).to(cuda)
    col = torch.from_numpy(g.colind).to(cuda).long()
    gen = torch.Generator(device=cuda).manual_seed(T)
    wide = torch.randn(g.ncols, 300, generator=gen, device=cuda, dtype=dtype)
    tol = REL_TOL if dtype == torch.float32 else 1e-13
    for k in WIDTHS:
        for off in (0, 1):  # off = 1: rows that start at no 16-byte boundary, odd row stride with [:, :299]
            X = wide[:, :299][:, off:off + k] if off else wide[:, :k].contiguous()
            want = torch.zeros(A.padded_rows(), k, dtype=torch.float64, device=cuda)
            want.index_add_(0, row, X.double()[col])
            scale = torch.zeros_like(want).index_add_(0, row, X.double().abs()[col]).clamp_min(1e-30)
            Y = A.spmm(X)
            assert float(((Y.double() - want).abs() / scale).max()) <= tol, (k, off)
            assert torch.equal(Y, A.spmm(X)), (k, off)
            big = torch.full((A.padded_rows(), k + 5), 3.0, device=cuda, dtype=dtype)
            A.spmm(X, big[:, 2:2 + k], accumulate=True)  # an unaligned Y between columns that stay
            err = (big[:, 2:2 + k].double() - 3.0 - want).abs() / (scale + 3.0)
            assert float(err.max()) <= tol, (k, off)
            assert bool((big[:, :2] == 3.0).all()) and bool((big[:, 2 + k:] == 3.0).all()), (k, off)
    A.close()
