"""Wrapped arrays whose tiles are filled only after they were wrapped: the dense-RHS product, whose plan
follows the set bits, takes the tiles as they are at its first call, and as they are at later ones."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_tiles_filled_after_wrapping(pkg, cuda, T):
    nb, nbc = 6, 120
    rp = torch.arange(nb + 1, dtype=torch.int32, device=cuda) * nbc
    ci = torch.arange(nbc, dtype=torch.int32, device=cuda).repeat(nb)
    tiles = torch.zeros(nb * nbc * T, dtype=pkg.word_dtype(T), device=cuda)
    A = pkg.B2SRMatrix.wrap(rp, ci, tiles, nb * T, nbc * T, T)
    full = {4: 15, 8: 255, 16: -1, 32: -1}[T]
    tiles.fill_(full)  # every bit
    X = torch.arange(1, 7, device=cuda, dtype=torch.float32).expand(nbc * T, 6).contiguous()
    want = np.tile(nbc * T * np.arange(1, 7, dtype=np.float32), (nb * T, 1))
    np.testing.assert_array_equal(A.spmm(X).cpu().numpy(), want)
    np.testing.assert_array_equal(A.transpose().spmm(X[: nb * T].contiguous()).cpu().numpy(),
                                  np.tile(nb * T * np.arange(1, 7, dtype=np.float32), (nbc * T, 1)))
    tiles[: nbc * T].zero_()  # the first tile-row empties again
    want[:T] = 0
    np.testing.assert_array_equal(A.spmm(X).cpu().numpy(), want)
    A.close()
