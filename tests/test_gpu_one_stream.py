"""Host threads that call one matrix on one stream: the kernels of a call (main, fix-up; classify, push,
gate) share the stream's scratch, so another thread's kernels may not come in between.  The threads are
native ones: Python's would hardly ever be inside the library together."""
from __future__ import annotations

import ctypes as C
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <pthread.h>
typedef int (*spmv_fn)(const void*, const void*, void*, int, void*);
typedef int (*spmm_fn)(const void*, const void*, int, long long, void*, long long, int, void*);
struct job { void* fn; const void* m; const void* x; char* y; long long step; int k, calls, bad; void* stream; pthread_barrier_t* b; };
static void* work(void* p) {
    struct job* j = (struct job*)p;
    for (int i = -1; i < j->calls; ++i) {
        if (i < 0) { pthread_barrier_wait(j->b); continue; }
        char* y = j->y + i * j->step;
        j->bad += 0 != (j->k ? ((spmm_fn)j->fn)(j->m, j->x, j->k, j->k, y, j->k, 0, j->stream)
                             : ((spmv_fn)j->fn)(j->m, j->x, y, 0, j->stream));
    }
    return 0;
}
int two_threads(void* fn, const void* m, const void* x0, const void* x1, void* y0, void* y1, long long step, int k, int calls,
                void* stream) {
    pthread_barrier_t b;
    pthread_barrier_init(&b, 0, 2);
    struct job j[2] = {{fn, m, x0, (char*)y0, step, k, calls, 0, stream, &b}, {fn, m, x1, (char*)y1, step, k, calls, 0, stream, &b}};
    pthread_t t[2];
    for (int i = 0; i < 2; ++i) pthread_create(&t[i], 0, work, &j[i]);
    for (int i = 0; i < 2; ++i) pthread_join(t[i], 0);
    return j[0].bad + j[1].bad;
}
"""


@pytest.fixture(scope="module")
def two_threads(tmp_path_factory):
    d = tmp_path_factory.mktemp("threads")
    (d / "t.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-pthread", "-o", str(d / "t.so"), str(d / "t.c")], check=True)
    fn = C.CDLL(str(d / "t.so")).two_threads
    fn.argtypes = [C.c_void_p] * 6 + [C.c_longlong, C.c_int, C.c_int, C.c_void_p]
    return fn


@pytest.mark.parametrize("T", [4, 32])
@pytest.mark.parametrize("what", ["spmm", "full", "pull", "push", "auto"])
def test_threads_on_one_stream(pkg, cuda, two_threads, what, T):
    lib, calls = pkg._lib.load(), 2000
    g = pkg.rmat(13, 16, seed=T)  # tile-rows of many tasks
    A = pkg.B2SRMatrix.from_graph(g, T, device=cuda)
    k = 3 if what == "spmm" else 0
    dtype = torch.float32 if what in ("spmm", "full") else torch.int32
    if dtype == torch.int32:
        A.set_launch("bin_bin_count", direction=what)
    fn = {"spmm": lib.b2sr_spmm_bin_full_full, "full": lib.b2sr_spmv_bin_full_full}.get(what, lib.b2sr_spmv_bin_bin_count)
    gen = torch.Generator().manual_seed(T)
    xs = []
    for share in (0.9, 0.02):  # counts: one over the direction lines, one under
        x = (torch.rand(g.ncols, generator=gen) < share).float().to(cuda)
        xs.append((x[:, None] * torch.arange(1, 4, device=cuda)).contiguous() if k else
                  A.pack_bits(x) if dtype == torch.int32 else x)
    call = A.spmm if k else A.spmv_bin_full_full if what == "full" else A.spmv_bin_bin_count
    want = [call(x).flatten() for x in xs]
    n = want[0].numel()
    ys = [torch.empty(calls, n, dtype=dtype, device=cuda) for _ in range(2)]
    torch.cuda.synchronize()
    rc = two_threads(C.cast(fn, C.c_void_p), A.handle, xs[0].data_ptr(), xs[1].data_ptr(), ys[0].data_ptr(),
                     ys[1].data_ptr(), 4 * n, k, calls, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    for i in range(2):
        bad = int((ys[i] != want[i]).any(dim=1).sum())
        assert bad == 0, f"{bad} of {calls} results of thread {i} wrong"
    A.close()
