"""Infinities and NaN in x and X reach exactly the rows that have a set column there: not through unset
columns of a tile, padding, the dense stages of long rows, pairwise sums or repeated slots."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import REL_TOL

pytestmark = pytest.mark.gpu


def _graph(pkg, T, n):
    """Rows of 0 to 30 entries over n + 3 columns, long rows, and full tiles beside single entries; n = 150000
    gives the more than 2^20 tiles from which T = 32 takes its form for large matrices."""
    rng = np.random.default_rng(T + n)
    rows, cols = [rng.integers(0, n, 9 * n)], [rng.integers(0, n + 3, 9 * n)]
    for r, m in ((7, 3000), (T + 1, 9000), (40 * T, 20000)):
        rows.append(np.full(m, r))
        cols.append(rng.choice(n + 3, m, replace=False))
    for tr in (60, 61):  # 300 full tiles in a row
        r, c = np.meshgrid(np.arange(tr * T, tr * T + T), np.arange(300 * T), indexing="ij")
        rows.append(r.ravel())
        cols.append(c.ravel())
    return pkg.from_edges(np.concatenate(rows), np.concatenate(cols), nrows=n, ncols=n + 3, drop_self_loops=False)


def _check(g, X, Y):
    """Every entry of Y against the row sums of X in 64 bits."""
    rows = np.repeat(np.arange(g.nrows), np.diff(g.rowptr))
    for k in range(X.shape[1]):
        x = X[g.colind, k]
        nan, pos, neg = (np.bincount(rows, m, g.nrows) > 0 for m in (np.isnan(x), x == np.inf, x == -np.inf))
        fin = np.where(np.isfinite(x), x, 0).astype(np.float64)
        want, scale = np.bincount(rows, fin, g.nrows), np.bincount(rows, np.abs(fin), g.nrows)
        y = Y[: g.nrows, k].astype(np.float64)
        bad = nan | (pos & neg)
        np.testing.assert_array_equal(np.isnan(y), bad)
        np.testing.assert_array_equal(y == np.inf, pos & ~bad)
        np.testing.assert_array_equal(y == -np.inf, neg & ~bad)
        ok = ~(bad | pos | neg)
        assert np.all(np.abs(y[ok] - want[ok]) <= REL_TOL * scale[ok])


def _values(rng, shape):
    x = rng.standard_normal(shape).astype(np.float32)
    r = rng.random(shape)
    for i, v in enumerate((np.nan, np.inf, -np.inf)):
        x[(r >= 0.004 * i) & (r < 0.004 * (i + 1))] = v
    return x


@pytest.mark.parametrize("T,n", [(4, 30000), (8, 30000), (16, 30000), (32, 30000), (32, 150000)])
def test_vector(pkg, cuda, T, n):
    g = _graph(pkg, T, n)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    assert (A.nblocks >= 1 << 20) == (n == 150000)
    x = _values(np.random.default_rng(T), (g.ncols, 1))
    for gather in ("auto", "ldg", "texture", "sparse"):
        A.set_launch("bin_full_full", gather=gather)
        y = A.spmv_bin_full_full(torch.from_numpy(x[:, 0].copy()).to(cuda))
        _check(g, x, y.cpu().numpy()[:, None])
    A.close()


@pytest.mark.parametrize("T", [4, 8, 16, 32])
@pytest.mark.parametrize("k", [1, 3, 40, 64, 130])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_dense_rhs(pkg, cuda, T, k, dtype):
    g = _graph(pkg, T, 25000)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    X = _values(np.random.default_rng(k), (g.ncols, k))
    Y = A.spmm(torch.from_numpy(X).to(cuda, dtype)).cpu().numpy()
    pick = sorted({0, k // 2, k - 1})
    _check(g, X[:, pick], Y[:, pick])
    A.close()
