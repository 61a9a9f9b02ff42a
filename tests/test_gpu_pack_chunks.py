"""The packer's chunks (b2sr_pack.cu) at their edges, bit-exact against the oracle: tile-rows around the
sizes of a chunk, rows of very different lengths, dense tiles and duplicates that overfill a chunk,
columns too many for 32-bit sort keys, and an unaligned tile array."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from gpu_util import to_np_words

pytestmark = pytest.mark.gpu


def _csr(rows, ncols):
    rowptr = np.zeros(len(rows) + 1, np.int32)
    rowptr[1:] = np.cumsum([len(r) for r in rows])
    return rowptr, np.concatenate([np.sort(np.asarray(r, np.int64)) for r in rows] + [[]]).astype(np.int32), ncols


def _shapes(T):
    rng = np.random.default_rng(T)
    pick = lambda n, hi: rng.choice(hi, n, replace=False)  # noqa: E731
    spread = [[] for _ in range(T)]  # one tile-row each, of 31 .. 1025 entries over its T rows
    edges = []
    for total in (0, 1, 31, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512, 513, 640, 641, 1025):
        cut = np.sort(rng.integers(0, total + 1, T - 1))
        edges += [pick(n, 90000) for n in np.diff(np.concatenate([[0], cut, [total]]))]
    yield "edges", _csr(edges, 90000)
    # a hub row beside short ones, and hubs whose entries are all at one end
    yield "uneven", _csr([pick(20000, 40000)] + [pick(7, 40000) for _ in range(2 * T)] + [np.arange(3000)]
                         + [np.arange(37000, 40000)] + spread[: T - 2] + [pick(900, 40000) for _ in range(T + 3)], 40000)
    # full tiles, and rows that repeat their columns
    yield "dense", _csr([np.arange(700)] * (T + 1), 700)
    yield "duplicates", _csr([np.repeat(pick(40, 5000), 30), np.full(2000, 17), pick(3, 5000)] * T, 5000)
    # tile-columns past 2^31 / T^2
    big = 1 << 30
    yield "wide", _csr([rng.integers(0, big, n) for n in rng.integers(0, 300, 3 * T)] + [[big - 1, big - 2]], big)


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_chunks_against_oracle(pkg, orc, cuda, T):
    for name, (rowptr, colind, ncols) in _shapes(T):
        nrows = len(rowptr) - 1
        A = pkg.B2SRMatrix.from_csr(rowptr, colind, nrows, ncols, T, device=cuda)
        brp, bci, tiles = A.download()
        wrp, wci, wtiles = orc.csr_to_b2sr(rowptr, colind, nrows, T)
        np.testing.assert_array_equal(brp, wrp, err_msg=name)
        np.testing.assert_array_equal(bci, wci, err_msg=name)
        np.testing.assert_array_equal(tiles, wtiles, err_msg=name)
        rows = np.repeat(np.arange(nrows), np.diff(rowptr)).astype(np.int64)
        assert A.nnz == np.unique(rows * ncols + colind).size, name
        A.close()


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_batch_into_an_unaligned_array(pkg, orc, cuda, T):
    """b2sr_ref_csr2bsr_batch writes tiles at any word address."""
    lib = pkg._lib.load()
    rowptr, colind, ncols = dict(_shapes(T))["edges"]
    nrows = len(rowptr) - 1
    wrp, wci, wtiles = orc.csr_to_b2sr(rowptr, colind, nrows, T)
    brp, bci = torch.from_numpy(wrp).to(cuda), torch.empty(len(wci), dtype=torch.int32, device=cuda)
    buf = torch.full((len(wtiles) + 2,), 5, dtype=pkg.word_dtype(T), device=cuda)
    rc = lib.b2sr_ref_csr2bsr_batch(rowptr.ctypes.data, colind.ctypes.data, nrows, ncols, len(colind), brp.data_ptr(),
                                    bci.data_ptr(), buf[1:].data_ptr(), T, len(wrp) - 1, len(wci))
    assert rc == 0
    got = to_np_words(buf, T)
    np.testing.assert_array_equal(bci.cpu().numpy(), wci)
    np.testing.assert_array_equal(got[1:-1], wtiles)
    assert got[0] == 5 and got[-1] == 5


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_transpose_digit_passes(pkg, orc, cuda, T):
    """One, two and three digit passes of the transpose's sort, with hub tile-columns; and wrapped tiles at an odd
    byte address, with bits set in the unused half of a T = 4 row."""
    rng = np.random.default_rng(T)
    for ncols in (400 * T, 200000 * T, 300000 * T):
        n, m = 600, 30000
        rows, cols = rng.integers(0, n, m), rng.integers(0, ncols, m)
        cols[: m // 3] = rng.integers(0, 5 * T, m // 3)
        g = pkg.from_edges(rows, cols, nrows=n, ncols=ncols, drop_self_loops=False)
        gt = pkg.from_edges(g.colind, np.repeat(np.arange(n), np.diff(g.rowptr)), nrows=ncols, ncols=n,
                            drop_self_loops=False)
        want = orc.csr_to_b2sr(gt.rowptr, gt.colind, ncols, T)
        A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
        for a, b in zip(A.transpose().download(), want):
            np.testing.assert_array_equal(a, b)
        rp, ci, tl = A.download()
        A.close()
        dirty = tl | 0x50 if T == 4 else tl
        buf = torch.zeros(dirty.size + 1, dtype=pkg.word_dtype(T), device=cuda)
        buf[1:] = torch.from_numpy(dirty.view(buf.cpu().numpy().dtype)).to(cuda)
        B = pkg.B2SRMatrix.wrap(torch.from_numpy(rp).to(cuda), torch.from_numpy(ci).to(cuda), buf[1:], n, ncols, T)
        for a, b in zip(B.transpose().download(), want):
            np.testing.assert_array_equal(a, b)
        B.close()


@pytest.mark.parametrize("T", [4, 8])
@pytest.mark.parametrize("ncols", [3000, 1 << 30])
def test_rows_that_are_merged(pkg, orc, cuda, T, ncols):
    """One tile-row per case of 129 to 512 entries: all in one row, runs of empty rows before, between
    and behind, single entries, rows before and behind each other's columns, and equal rows."""
    rng = np.random.default_rng(T + ncols)
    pick = lambda n: rng.choice(min(ncols, 1 << 20), n, replace=False)  # noqa: E731
    rows = []
    for n in (129, 255, 256, 257, 500, 512):
        for at in (0, 1, T - 2, T - 1):  # (others, their sizes) beside one long row
            for rest in (0, 1):
                tr = [pick(rest) for _ in range(T)]
                tr[at] = pick(n - rest * (T - 1))
                rows += tr
        cut = np.linspace(0, n, T + 1).astype(int)
        rows += [np.arange(cut[r], cut[r + 1]) for r in range(T)]  # ascending from row to row
        rows += [np.arange(cut[T - 1 - r], cut[T - r]) for r in range(T)]
        rows += [np.arange(n // T) * 5] * T
        rows += [pick(n // 2), pick(n - n // 2)] + [[] for _ in range(T - 2)]
        rows += [[] for _ in range(T - 2)] + [pick(n // 2), pick(n - n // 2)]
    rowptr, colind, _ = _csr(rows, ncols)
    A = pkg.B2SRMatrix.from_csr(rowptr, colind, len(rows), ncols, T, device=cuda)
    for got, want in zip(A.download(), orc.csr_to_b2sr(rowptr, colind, len(rows), T)):
        np.testing.assert_array_equal(got, want)
    A.close()
