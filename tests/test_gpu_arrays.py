"""Where a matrix's arrays live: blocks of cudaMalloc that other processes and devices can open; reused by
later matrices of about their size, and given back by b2sr_trim."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def describe(pkg, A):
    d = pkg._lib.MatrixDesc()
    assert pkg._lib.load().b2sr_matrix_describe(A.handle, C.byref(d)) == 0
    return d


@pytest.mark.parametrize("T", [4, 32])
def test_arrays_can_be_exported(pkg, cuda, tmp_path, T):
    cu = C.CDLL("libcuda.so.1")
    A = pkg.B2SRMatrix.from_graph(pkg.rmat(11, 8, seed=T), T, device=cuda)
    A.save(tmp_path / "m.b2sr")
    L = pkg.B2SRMatrix.load(tmp_path / "m.b2sr", device=cuda)
    for M in (A, A.transpose(), L):
        d = describe(pkg, M)
        for p, n in ((d.d_rowptr, 4 * (d.nblockrows + 1)), (d.d_colind, 4 * d.nblocks), (d.d_tiles, d.nblocks * T * max(T // 8, 1))):
            handle, base, size = (C.c_char * 64)(), C.c_uint64(), C.c_size_t()
            assert cu.cuIpcGetMemHandle(handle, C.c_uint64(p)) == 0
            assert cu.cuMemGetAddressRange_v2(C.byref(base), C.byref(size), C.c_uint64(p)) == 0
            assert base.value == p and size.value >= n
    L.close()
    A.close()


def free_bytes():
    """Free bytes on the device."""
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_a_graph_per_step_takes_no_more_memory(pkg, cuda):
    """Graphs of slightly different sizes, packed, transposed, multiplied and freed: the memory of the
    second step serves the twentieth."""
    rng = np.random.default_rng(3)
    for step in range(20):
        n = 60000 + int(rng.integers(0, 3000))
        g = pkg.erdos_renyi(n, 10.0, seed=step)
        A = pkg.B2SRMatrix.from_graph(g, 16, device=cuda)
        X = torch.ones(A.padded_rows(), 4, device=cuda)
        assert float(A.spmm(X).sum()) == 4.0 * g.nnz and float(A.transpose().spmm(X).sum()) == 4.0 * g.nnz
        A.close()
        if step == 2:
            free = free_bytes()
    assert free - free_bytes() <= 32 << 20  # two of the arrays' 19 MB; twenty steps that kept theirs would hold 900 MB


def test_trim_gives_back(pkg, cuda):
    """200 MB of tiles: kept when freed, gone after a trim; and more small matrices than blocks are kept."""
    lib = pkg._lib.load()
    g = pkg.erdos_renyi(200000, 8.0, seed=2)
    lib.b2sr_trim()
    empty = free_bytes()
    A = pkg.B2SRMatrix.from_graph(g, 32, device=cuda)
    tiles = A.nblocks * 128
    assert tiles > 150 << 20
    A.close()
    assert empty - free_bytes() >= tiles
    lib.b2sr_trim()
    assert empty - free_bytes() <= 8 << 20
    after = []
    for _ in range(2):  # the first time also loads the kernels
        many = [pkg.B2SRMatrix.from_graph(pkg.erdos_renyi(100 + i, 3.0, seed=i), 8, device=cuda) for i in range(400)]
        for i, M in enumerate(many):
            y = M.spmv_bin_full_full(torch.ones(M.ncols, device=cuda))
            np.testing.assert_array_equal(y.cpu().numpy()[: M.nrows], pkg.erdos_renyi(100 + i, 3.0, seed=i).degrees())
            M.close()
        lib.b2sr_trim()
        after.append(free_bytes())
    assert after[0] - after[1] <= 8 << 20
