"""No block goes back to the allocator while a kernel can still use it: an allocator hook that looks, at
each free, whether the work queued before it has ended, with failures at every allocation of a call."""
from __future__ import annotations

import contextlib
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


class Hook:
    """b2sr_set_allocator hooks over torch's allocator.  fail_at: the allocation that fails, counted from
    now; busy: frees made while the stream had work in flight."""

    def __init__(self, L):
        self.blocks, self.n, self.fail_at, self.busy, self.freed, self.stream = {}, 0, -1, 0, 0, None

        def alloc(nbytes, _ctx):
            self.n += 1
            if self.n == self.fail_at:
                return None
            t = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            self.blocks[t.data_ptr()] = t
            return t.data_ptr()

        def free(ptr, _ctx):
            self.freed += 1
            if self.stream is not None and not self.stream.query():
                self.busy += 1
            self.blocks.pop(ptr)

        self.alloc, self.free = L.ALLOC_FN(alloc), L.FREE_FN(free)


@contextlib.contextmanager
def hooked(pkg):
    L = pkg._lib
    h = Hook(L)
    L.load().b2sr_set_allocator(h.alloc, h.free, None)
    try:
        yield h
    finally:
        L.load().b2sr_set_allocator(L.ALLOC_FN(), L.FREE_FN(), None)


def queue_work():
    torch.cuda._sleep(20_000_000)  # about 10 ms on the stream


@pytest.mark.parametrize("T", [4, 8, 16, 32])
def test_first_spmm_with_failing_allocations(pkg, cuda, T):
    g = pkg.rmat(11, 16, seed=T)
    X = torch.ones(g.ncols, 8, device=cuda)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with hooked(pkg) as h, torch.cuda.stream(s):
        fail = 0
        while True:
            fail += 1
            A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
            Y = torch.empty(A.padded_rows(), 8, device=cuda)
            s.synchronize()
            h.stream, h.n, h.fail_at = s, 0, fail
            queue_work()
            rc = pkg._lib.load().b2sr_spmm_bin_full_full(A.handle, X.data_ptr(), 8, 8, Y.data_ptr(), 8, 0, s.cuda_stream)
            reached, h.fail_at = h.n >= fail, -1
            assert rc == (3 if reached else 0), (fail, rc)
            assert h.busy == 0, f"block freed in use when allocation {fail} fails"
            h.stream = None
            A.close()
            assert not h.blocks
            if not reached:
                break
        assert fail > (4 if T >= 8 else 3)  # every allocation of the call has failed once
        # the library goes on as if nothing had happened
        A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
        assert torch.equal(A.spmm(X)[: g.nrows, 0].cpu(), torch.from_numpy(g.degrees()).float())
        A.close()


@pytest.mark.parametrize("T", [4, 32])
def test_transpose_of_an_empty_matrix_is_complete(pkg, cuda, T):
    """The cached transpose may be used on any stream, and freed by the caller that lost the race to build
    it, so its arrays are written when the call returns."""
    A = pkg.B2SRMatrix.from_graph(pkg.from_edges([], [], nrows=500, ncols=300), T, device=cuda)
    s = torch.cuda.Stream()
    out = C.c_void_p()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        queue_work()
        rc = pkg._lib.load().b2sr_matrix_transpose(A.handle, s.cuda_stream, C.byref(out))
        done = s.query()
    assert rc == 0 and done
    At = A.transpose()
    assert (At.nrows, At.ncols, At.nblocks) == (300, 500, 0) and not At.download()[0].any()
    A.close()


@pytest.mark.parametrize("later", ["free", "trim"])
def test_free_during_a_capture_keeps_the_memory(pkg, cuda, later):
    """The device cannot be waited for while a stream is being captured, so nothing goes back to the
    allocator until a later call can."""
    cu, lib = C.CDLL("libcuda.so.1"), pkg._lib.load()
    g = pkg.erdos_renyi(2000, 8.0, seed=1)
    s = torch.cuda.Stream()
    with hooked(pkg) as h:
        A, B = pkg.B2SRMatrix.from_graph(g, 8, device=cuda), pkg.B2SRMatrix.from_graph(g, 8, device=cuda)
        A.spmm(torch.ones(g.ncols, 8, device=cuda))
        torch.cuda.synchronize()
        held, h.freed = len(h.blocks), 0
        assert cu.cuStreamBeginCapture_v2(C.c_void_p(s.cuda_stream), 0) == 0
        A.close()
        freed, graph = h.freed, C.c_void_p()
        cu.cuStreamEndCapture(C.c_void_p(s.cuda_stream), C.byref(graph))  # invalidated: an error, no graph
        assert freed == 0 and len(h.blocks) == held
        torch.cuda.synchronize()
        B.close() if later == "free" else lib.b2sr_trim()
        assert h.freed > 0
        B.close()
        assert not h.blocks


def test_a_free_hook_may_free_another_matrix(pkg, cuda):
    """As Python's garbage collector does, when it runs inside the hook."""
    g = pkg.erdos_renyi(1000, 4.0, seed=1)
    with hooked(pkg) as h:
        A, B = pkg.B2SRMatrix.from_graph(g, 8, device=cuda), pkg.B2SRMatrix.from_graph(g, 4, device=cuda)
        others = [B]

        class Blocks(dict):
            def pop(self, ptr):
                if others:
                    others.pop().close()
                return super().pop(ptr)

        h.blocks = Blocks(h.blocks)
        A.close()
        assert not h.blocks
