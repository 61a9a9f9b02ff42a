"""A CSR whose arrays are shorter than the entry count that comes with it: refused by its row pointer, and
no column is read."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_entry_count_past_the_arrays(pkg, cuda, T):
    lib, out = pkg._lib.load(), C.c_void_p()
    rp = torch.tensor([0, 2, 3, 3, 4], dtype=torch.int32, device=cuda)
    ci = torch.tensor([0, 3, 1, 2], dtype=torch.int32, device=cuda)
    for nnz in (5, 100, 1 << 24, (1 << 24) + 3):
        assert lib.b2sr_pack_csr(rp.data_ptr(), ci.data_ptr(), 4, 4, nnz, T, None, C.byref(out)) == 2
        assert out.value is None
    A = pkg.B2SRMatrix.from_csr(rp.cpu().numpy(), ci.cpu().numpy(), 4, 4, T, device=cuda)
    np.testing.assert_array_equal(A.spmv_bin_full_full(torch.ones(4, device=cuda)).cpu().numpy()[:4], [2, 1, 0, 1])
    A.close()
