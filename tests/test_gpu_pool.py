"""The library's device memory: matrices made and freed over and over reuse their memory and keep the
amount they hold bounded; other streams and threads get blocks that nothing uses any more."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_memory_is_bounded_and_given_back(pkg, cuda):
    g = pkg.rmat(15, 16, seed=4)
    lib = pkg._lib.load()
    torch.cuda.synchronize()
    lib.b2sr_trim()
    free0, total = torch.cuda.mem_get_info()
    for _ in range(20):
        A = pkg.B2SRMatrix.from_graph(g, 8, device=cuda)
        A.transpose()
        A.spmm(torch.ones(g.ncols, 8, device=cuda))
        A.close()
    torch.cuda.synchronize()
    held = free0 - torch.cuda.mem_get_info()[0]
    assert held <= total // 256 + (64 << 20)  # + what torch and the context took in between
    lib.b2sr_trim()
    after = free0 - torch.cuda.mem_get_info()[0]
    assert after <= held


@pytest.mark.parametrize("T", [4, 32])
def test_reused_memory_on_two_threads(pkg, orc, cuda, T):
    """Two threads pack, multiply and free different graphs on their own streams."""
    errors = []

    def work(seed):
        try:
            stream = torch.cuda.Stream()
            rng = np.random.default_rng(seed)
            with torch.cuda.stream(stream):
                for i in range(15):
                    g = pkg.erdos_renyi(int(rng.integers(500, 6000)), 9.0, seed=seed * 100 + i)
                    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
                    y = A.spmv_bin_full_full(torch.ones(g.ncols, device=cuda))
                    dy = A.transpose().spmv_bin_full_full(torch.ones(A.padded_rows(), device=cuda))
                    want = g.degrees().astype(np.float32)
                    got, got_t = y.cpu().numpy()[: g.nrows], dy.cpu().numpy()[: g.nrows]
                    A.close()
                    if not (np.array_equal(got, want) and np.array_equal(got_t, want)):
                        errors.append((seed, i))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append((seed, repr(e)))

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
