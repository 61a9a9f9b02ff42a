"""The multiplies that spread a 16 x 16 or 32 x 32 tile over lanes (b2sr_widetile.cuh) against
the oracle: staged long rows with sparse and dense stages, ragged ends, every short-row bin,
and frontiers on both sides of the mostly-zero rule."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_util import REL_TOL, from_np_words, full_full_error, to_np_words

pytestmark = pytest.mark.gpu


def _mixed(pkg, n, degree, seed):
    """An ER graph with a dense block, a hub row, and tile-rows of 0, 1, 2, ... 40 tiles at its end."""
    rng = np.random.default_rng(seed)
    top = n - 32 * 41
    m = int(top * degree)
    rows = [rng.integers(32, top, m), np.repeat(np.arange(64, 200), 700), np.full(n // 3, 40)]
    cols = [rng.integers(0, n, m), np.tile(np.arange(5, 705), 136), rng.integers(0, n, n // 3)]
    for t in range(41):  # tile-row t of the tail: t tiles at T = 32, one to a few bits each
        c = np.repeat(np.arange(t) * 97 % (n // 32) * 32, 3)
        rows.append(rng.integers(top + 32 * t, top + 32 * t + 32, c.size))
        cols.append(np.minimum(c + rng.integers(0, 32, c.size), n - 1))
    return pkg.from_edges(np.concatenate(rows), np.minimum(np.concatenate(cols), n - 8), nrows=n, ncols=n - 7,
                          drop_self_loops=False)


# more tiles at T = 32 than the FP32 form's threshold (2^20), and fewer
@pytest.mark.parametrize("n,degree", [(70003, 20.0), (9001, 12.0)])
def test_full_full_t32(pkg, orc, cuda, n, degree):
    rng = np.random.default_rng(3)
    g = _mixed(pkg, n, degree, 5)
    A = pkg.B2SRMatrix.from_graph(g, 32, device=cuda)
    assert (A.nblocks >= 1 << 20) == (n > 20000)
    x = rng.standard_normal(g.ncols).astype(np.float32)
    xd = torch.from_numpy(x).to(cuda)
    y = A.spmv_bin_full_full(xd)
    assert full_full_error(orc, g, x, y.cpu().numpy()) <= REL_TOL
    assert torch.equal(y, A.spmv_bin_full_full(xd))
    assert bool((y[g.nrows:] == 0).all())
    y0 = torch.from_numpy(rng.standard_normal(A.padded_rows()).astype(np.float32)).to(cuda)
    ya = y0.clone()
    A.spmv_bin_full_full(xd, ya, accumulate=True)
    assert torch.equal(ya, y0 + y)
    ones = A.spmv_bin_full_full(torch.ones(g.ncols, device=cuda)).cpu().numpy()
    np.testing.assert_array_equal(ones[: g.nrows], g.degrees().astype(np.float32))
    A.close()


@pytest.mark.parametrize("density", [0.0, 0.004, 0.02, 0.5, 1.0])
def test_bits_t32(pkg, orc, cuda, density):
    g = _mixed(pkg, 9001, 12.0, 6)
    A = pkg.B2SRMatrix.from_graph(g, 32, device=cuda)
    brp, bci, tiles = orc.csr_to_b2sr(g.rowptr, g.colind, g.nrows, 32)
    rng = np.random.default_rng(int(density * 1000))
    on = np.zeros(A.nblockcols * 32, np.float32)
    on[: g.ncols] = rng.random(g.ncols) < density
    xb = orc.pack_vec_bits(on, 32)
    xt = from_np_words(xb, 32, cuda)
    mask = orc.pack_vec_bits((rng.random(A.padded_rows()) < 0.5).astype(np.float32), 32)
    np.testing.assert_array_equal(to_np_words(A.spmv_bin_bin_bin(xt), 32), orc.bmv_bin_bin_bin(32, brp, bci, tiles, xb))
    np.testing.assert_array_equal(to_np_words(A.spmv_bin_bin_bin_masked(xt, from_np_words(mask, 32, cuda)), 32),
                                  orc.bmv_bin_bin_bin_masked(32, brp, bci, tiles, xb, mask))
    cnt = orc.bmv_bin_bin_count(32, brp, bci, tiles, xb)
    np.testing.assert_array_equal(A.spmv_bin_bin_count(xt).cpu().numpy(), cnt)
    np.testing.assert_array_equal(A.spmv_bin_bin_full(xt).cpu().numpy(), cnt.astype(np.float32))
    A.close()


@pytest.mark.parametrize("T", [16, 32])
@pytest.mark.parametrize("bits", [32, 64])
def test_multi_frontier(pkg, cuda, T, bits):
    """Column by column against the FP32 multiply of the same matrix: bit f of y[v] is set where it is not zero."""
    g = _mixed(pkg, 5003, 9.0, 7)
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    dt = torch.int32 if bits == 32 else torch.int64
    gen = torch.Generator(device=cuda).manual_seed(bits + T)
    on = torch.rand(g.ncols, bits, generator=gen, device=cuda) < 0.003
    seen = torch.rand(A.padded_rows(), bits, generator=gen, device=cuda) < 0.2
    shift = torch.arange(bits, device=cuda)
    words = lambda b: (b.long() << shift).sum(1).to(dt)  # noqa: E731
    want = A.spmm(on.float()) != 0
    assert torch.equal(A.spmv_multi_bits(words(on)), words(want))
    assert torch.equal(A.spmv_multi_bits(words(on), mask=words(seen)), words(want & ~seen))
    y = words(seen)
    A.spmv_multi_bits(words(on), y, accumulate=True)
    assert torch.equal(y, words(want | seen))
    A.close()
