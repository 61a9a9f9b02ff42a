"""The work that a user of this library has it do, as cases that can be timed and compared.

A case is a dict of plain values; `op` says which program it is:

  full       y = A.x, FP32 x and y (B2SRMatrix.spmv_bin_full_full): PageRank-like iterations, neighbour sums
  bits       y = A.x over bits, AND NOT a visited mask where `masked` (one BFS step)
  count      neighbour counts of a marked vertex set: int32, or FP32 where `as_float`
  bfs        a breadth-first search from one vertex: `levels` masked steps and the visited update between them
  multi      32 or 64 frontiers per step, one bit of a word each, with the visited sets as the mask
  spmm       Y = A.X, dense features X [ncols, k], FP32 or FP64
  train      one forward and backward of the sum aggregation through autograd, on a kept matrix
  newgraph   the same on a graph that is new in each pass (a sampled mini-batch): packing, plans and transpose count
  pack       CSR on the device -> B2SR on the device

Graphs (`graph`): "rmat" (2^scale vertices, 16 edges a vertex, a = .57, b = c = .19, symmetric), "er" (symmetric
Erdos-Renyi, n vertices), "rect" (bipartite block, n x ncols), "batch" (`count` ER graphs of uneven sizes stacked
block-diagonally, offsets multiples of 32).  All have sorted rows without duplicates or self-loops.
"""
import json
import math

import torch

import __graft_entry__ as entry

pkg = entry.load_package()

EDGE_FACTOR = 16
BATCH_N = (64, 65536)     # vertices of one graph of a batch, log-uniform
BATCH_DEGREE = (4.0, 32.0)


# ---- graphs ---------------------------------------------------------------------------------
def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def generator(seed):
    g = torch.Generator(device=device())
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def to_csr(rows, cols, nrows, ncols):
    """Sorted, duplicate-free CSR (int32) of the given entries."""
    key = torch.unique(rows * ncols + cols)
    r = key // ncols
    rowptr = torch.zeros(nrows + 1, dtype=torch.int32, device=key.device)
    rowptr[1:] = torch.cumsum(torch.bincount(r, minlength=nrows), 0)
    return rowptr, (key - r * ncols).to(torch.int32)


def symmetric_csr(u, v, n):
    keep = u != v
    u, v = u[keep], v[keep]
    return to_csr(torch.cat([u, v]), torch.cat([v, u]), n, n)


def integers(high, count, gen):
    return torch.randint(int(high), (int(count),), generator=gen, device=device())


def relabelled(case, graph, seed):
    """The graph with its blocks of 32 vertices in another order, so that the packed arrays' lengths stay the same.

    R-MAT by flipping bits of the labels (quadrants swapped at some levels), the others by a random order."""
    rowptr, colind, nrows, ncols = graph
    gen, dev = generator(seed), rowptr.device
    rows = torch.repeat_interleave(torch.arange(nrows, device=dev), (rowptr[1:] - rowptr[:-1]).long())
    if case["graph"] == "rmat":
        flip = int(integers(nrows // 32, 1, gen)) * 32
        return (*to_csr(rows ^ flip, colind.long() ^ flip, nrows, ncols), nrows, ncols)

    def order(n):  # new label of every vertex; a last block of fewer than 32 stays where it is
        first = torch.arange(n, device=dev)
        full = n // 32
        first[: full * 32] += ((torch.randperm(full, generator=gen, device=dev) - torch.arange(full, device=dev)) * 32
                               ).repeat_interleave(32)
        return first

    new_row = order(nrows)
    new_col = order(ncols) if case["graph"] == "rect" else new_row
    return (*to_csr(new_row[rows], new_col[colind.long()], nrows, ncols), nrows, ncols)


def make_graph(case, seed):
    """(rowptr, colind, nrows, ncols) on the device."""
    if case["op"] == "pack":
        return relabelled(case, make_graph({**case, "op": ""}, 17), seed)
    gen, dev = generator(seed), device()
    kind = case["graph"]
    if kind == "rmat":
        n = 1 << case["scale"]
        m = EDGE_FACTOR * n
        u = torch.zeros(m, dtype=torch.int64, device=dev)
        v = torch.zeros(m, dtype=torch.int64, device=dev)
        for _ in range(case["scale"]):
            r = torch.rand(m, generator=gen, device=dev)
            u = 2 * u + (r >= 0.76)
            v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        return (*symmetric_csr(u, v, n), n, n)
    if kind == "er":
        n = case["n"]
        m = int(n * case["degree"] / 2)
        return (*symmetric_csr(integers(n, m, gen), integers(n, m, gen), n), n, n)
    if kind == "rect":
        n, nc = case["n"], case["ncols"]
        m = int(n * case["degree"])
        return (*to_csr(integers(n, m, gen), integers(nc, m, gen), n, nc), n, nc)
    assert kind == "batch", kind
    lo, hi = BATCH_N
    # the quantiles of the log-uniform sizes in a random order: every batch of a count has as many vertices
    q = (torch.randperm(case["count"], generator=gen, device=dev) + 0.5) / case["count"]
    sizes = torch.exp(math.log(lo) + q.double() * (math.log(hi) - math.log(lo))).to(torch.int64)
    degree = torch.rand(case["count"], generator=gen, device=dev, dtype=torch.float64)
    degree = BATCH_DEGREE[0] + degree * (BATCH_DEGREE[1] - BATCH_DEGREE[0])
    ends = torch.cumsum((sizes + 31) // 32 * 32, 0)
    n = int(ends[-1])
    edges = (sizes * degree / 2).to(torch.int64)
    which = torch.repeat_interleave(torch.arange(case["count"], device=dev), edges)
    size, start = sizes[which], (ends - (sizes + 31) // 32 * 32)[which]
    ab = torch.rand(2, which.numel(), generator=gen, device=dev, dtype=torch.float64)
    u, v = (torch.minimum((ab[i] * size).to(torch.int64), size - 1) + start for i in (0, 1))
    return (*symmetric_csr(u, v, n), n, n)


def pack_words(mask, T):
    """Bit words of a boolean vector, MSB first, as the library lays them out (plain torch)."""
    n = mask.numel()
    padded = torch.zeros((n + T - 1) // T * T, dtype=torch.int64, device=mask.device)
    padded[:n] = mask
    w = (padded.view(-1, T) << torch.arange(T - 1, -1, -1, device=mask.device)).sum(1)
    if T > 8:
        w = torch.where(w >= 1 << (T - 1), w - (1 << T), w)  # the signed word of the same bits
    return w.to(pkg.word_dtype(T))


def padded_rows(case, n):
    return (n + case["T"] - 1) // case["T"] * case["T"]


# ---- inputs ---------------------------------------------------------------------------------
def make_inputs(case, seed):
    """The call's inputs beside the matrix, as plain tensors."""
    rowptr, colind, nrows, ncols = make_graph(case, seed)
    s = {"case": case, "rowptr": rowptr, "colind": colind, "nrows": nrows, "ncols": ncols}
    gen, dev = generator(seed + 7919), device()
    op, T = case["op"], case["T"]
    if op == "full":
        s["x"] = torch.rand(ncols, generator=gen, device=dev)
    elif op in ("bits", "count"):
        s["on"] = torch.rand(ncols, generator=gen, device=dev) < case["density"]
        s["x"] = pack_words(s["on"], T)
        if case.get("masked"):
            s["mask"] = pack_words(torch.rand(padded_rows(case, nrows), generator=gen, device=dev) < 0.5, T)
    elif op == "bfs":
        degree = rowptr[1:] - rowptr[:-1]
        ok = torch.nonzero(degree > 0).flatten()
        start = torch.zeros(ncols, dtype=torch.bool, device=dev)
        start[ok[int(integers(ok.numel(), 1, gen))]] = True
        s["x"] = pack_words(start, T)
    elif op == "multi":
        dt = torch.int32 if case["word_bits"] == 32 else torch.int64
        x = torch.zeros(ncols, dtype=torch.int64, device=dev)
        seen = torch.zeros(padded_rows(case, nrows), dtype=torch.int64, device=dev)
        for f in range(case["word_bits"]):
            # each frontier's density is drawn from 0.1% to 5%
            d = 10 ** (-3 + 1.7 * float(torch.rand(1, generator=gen, device=dev)))
            x |= (torch.rand(ncols, generator=gen, device=dev) < d).to(torch.int64) << f
            seen |= (torch.rand(seen.numel(), generator=gen, device=dev) < 4 * d).to(torch.int64) << f
        s["x"], s["mask"] = x.to(dt), seen.to(dt)
    elif op in ("spmm", "train", "newgraph"):
        dt = torch.float64 if case.get("fp64") else torch.float32
        s["x"] = torch.randn(ncols, case["k"], generator=gen, device=dev, dtype=dt)
        if op != "spmm":
            s["dy"] = torch.randn(nrows, case["k"], generator=gen, device=dev, dtype=dt)
    return s


def prepare(case, seed):
    s = make_inputs(case, seed)
    if case["op"] not in ("newgraph", "pack"):
        A = pkg.B2SRMatrix.from_csr(s["rowptr"], s["colind"], s["nrows"], s["ncols"], case["T"])
        if case.get("direction") == "auto":
            A.set_launch("bin_bin_bin", direction="auto")
            A.transpose()
        s["A"] = A
        del s["rowptr"], s["colind"]  # the packed form is what such a program keeps
    if case["op"] in ("train", "newgraph"):
        s["x"].requires_grad_(True)
    return s


class DeviceArray:
    """An array of a packed matrix, for torch.as_tensor: the tensor holds this object, and it the matrix."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": typestr, "version": 3}


def packed_arrays(A):
    """(rowptr, colind, tiles) of a packed matrix, as tensors over its own arrays."""
    d = pkg._lib.MatrixDesc()
    pkg._lib.check(pkg._lib.load().b2sr_matrix_describe(A.handle, d), "b2sr_matrix_describe")
    word = {4: "|u1", 8: "|u1", 16: "<i2", 32: "<i4"}[A.tile_dim]
    return tuple(torch.as_tensor(DeviceArray(A, p, n, t), device="cuda") for p, n, t in
                 ((d.d_rowptr, d.nblockrows + 1, "<i4"), (d.d_colind, d.nblocks, "<i4"),
                  (d.d_tiles, d.nblocks * A.tile_dim, word)))


def step(A, s):
    """Forward and backward of the aggregation; the outputs are Y and dX."""
    y = pkg.aggregate(A, s["x"])
    (dx,) = torch.autograd.grad(y, s["x"], s["dy"])
    return y.detach(), dx


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "pack":
        return packed_arrays(
            pkg.B2SRMatrix.from_csr(state["rowptr"], state["colind"], state["nrows"], state["ncols"], case["T"]))
    if op == "newgraph":
        A = pkg.B2SRMatrix.from_csr(state["rowptr"], state["colind"], state["nrows"], state["ncols"], case["T"])
        return step(A, state)
    A, x = state["A"], state["x"]
    if op == "full":
        return A.spmv_bin_full_full(x)
    if op == "bits":
        return A.spmv_bin_bin_bin_masked(x, state["mask"]) if case.get("masked") else A.spmv_bin_bin_bin(x)
    if op == "count":
        return A.spmv_bin_bin_full(x) if case.get("as_float") else A.spmv_bin_bin_count(x)
    if op == "multi":
        return A.spmv_multi_bits(x, mask=state["mask"])
    if op == "spmm":
        return A.spmm(x)
    if op == "train":
        return step(A, state)
    assert op == "bfs", op
    visited, frontier, levels = x, x, []
    for _ in range(case["levels"]):
        frontier = A.spmv_bin_bin_bin_masked(frontier, visited)
        visited = visited | frontier
        levels.append(frontier)
    return {"visited": visited, "levels": levels}


# ---- what a pass cannot do without ------------------------------------------------------------
_work = {}


def work(case):
    """Bytes and operations of one pass, counted on a graph of the case's kind (its sizes hardly depend on the seed)."""
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _work:
        _work[key] = _count(case)
    return _work[key]


def _count(case):
    op, T = case["op"], case["T"]
    rowptr, colind, n, nc = make_graph(case, 1)
    nnz = colind.numel()
    rows = torch.repeat_interleave(torch.arange(n, device=rowptr.device), (rowptr[1:] - rowptr[:-1]).long())
    nb, nbc = -(-n // T), -(-nc // T)
    nt = torch.unique((rows // T) * nbc + colind // T).numel()
    wb = 1 if T <= 8 else T // 8
    matrix = 4 * (nb + 1) + (4 + T * wb) * nt
    if op == "full":
        return {"bytes": matrix + 4 * nc + 4 * nb * T, "flops": nnz}
    if op in ("bits", "bfs"):
        # BFS: the matrix once, the frontier that each level writes, the visited set
        vectors = case["levels"] + 2 if op == "bfs" else 3 if case.get("masked") else 2
        return {"bytes": matrix + vectors * wb * max(nb, nbc), "flops": nnz}
    if op == "count":
        return {"bytes": matrix + wb * nbc + 4 * nb * T, "flops": nnz}
    if op == "multi":
        return {"bytes": matrix + case["word_bits"] // 8 * (nc + 2 * nb * T), "flops": nnz}
    if op == "pack":
        return {"bytes": 4 * (n + 1 + nnz) + matrix, "flops": nnz}
    elem = 8 if case.get("fp64") else 4
    if op == "spmm":
        return {"bytes": matrix + elem * case["k"] * (nc + nb * T), "flops": nnz * case["k"]}
    matrices = 2 * matrix if op == "train" else 4 * (n + 1 + nnz) + 2 * matrix
    return {"bytes": matrices + elem * case["k"] * 2 * (n + nc), "flops": 2 * nnz * case["k"]}


# ---- the same in 64 bits, plain torch -----------------------------------------------------------
def exact(case, seed):
    op = case["op"]
    if op not in ("full", "spmm", "train", "newgraph") and not (op == "count" and case.get("as_float")):
        return None  # whole numbers
    s = make_inputs(case, seed)
    n, nc = s["nrows"], s["ncols"]
    rowptr, colind = s["rowptr"].long(), s["colind"].long()

    def product(rp, ci, rows_, cols_, x, out_rows):
        a = torch.sparse_csr_tensor(rp, ci, torch.ones(ci.numel(), dtype=torch.float64, device=ci.device), (rows_, cols_))
        x = x.double()
        y = torch.zeros(out_rows, x.shape[1], dtype=torch.float64, device=ci.device)
        y[:rows_] = a @ x
        return y

    if op == "full":
        return product(rowptr, colind, n, nc, s["x"][:, None], padded_rows(case, n))[:, 0]
    if op == "count":
        return product(rowptr, colind, n, nc, s["on"][:, None], padded_rows(case, n))[:, 0]
    if op == "spmm":
        return product(rowptr, colind, n, nc, s["x"], padded_rows(case, n))
    rows = torch.repeat_interleave(torch.arange(n, device=rowptr.device), rowptr[1:] - rowptr[:-1])
    rp_t, ci_t = to_csr(colind, rows, nc, n)
    return (product(rowptr, colind, n, nc, s["x"], n), product(rp_t.long(), ci_t.long(), nc, n, s["dy"], nc))


# ---- the cases ------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest: a neighbour sum on a 4096-vertex graph, where the call's own latency is all there is
        dict(name="full_er4096_t8", op="full", graph="er", n=4096, degree=16.0, T=8),
        # the library's headline multiply, and the largest tile of its tile sweep
        dict(name="full_rmat20_t4", op="full", graph="rmat", scale=20, T=4),
        dict(name="full_rmat20_t32", op="full", graph="rmat", scale=20, T=32),
        # one step of a BFS with a sparse frontier
        dict(name="bits_rmat20_t4", op="bits", graph="rmat", scale=20, T=4, density=0.01, masked=False),
        # how many neighbours are in a large marked set (label counts, k-core, triangle prefilters)
        dict(name="count_rmat20_t16", op="count", graph="rmat", scale=20, T=16, density=0.3, as_float=False),
        # a whole BFS: many short steps, frontiers from one vertex to half the graph, direction chosen by the library
        dict(name="bfs_rmat18_t8", op="bfs", graph="rmat", scale=18, T=8, levels=5, direction="auto"),
        # multi-source BFS step (betweenness, landmarks)
        dict(name="multi64_rmat18_t4", op="multi", graph="rmat", scale=18, T=4, word_bits=64),
        # feature aggregation with sizes that are multiples of nothing
        dict(name="spmm_er100003_k50_t8", op="spmm", graph="er", n=100003, degree=11.0, T=8, k=50),
        # inference on a batch of 512 uneven graphs in one launch
        dict(name="spmm_batch512_k64_t4", op="spmm", graph="batch", count=512, T=4, k=64),
        # full-graph training: forward and backward of one aggregation
        dict(name="train_rmat20_k128_t4", op="train", graph="rmat", scale=20, T=4, k=128),
        # mini-batch training: every step has its own sampled graph
        dict(name="newgraph_rmat16_k32_t8", op="newgraph", graph="rmat", scale=16, T=8, k=32),
        # conversion of a large graph
        dict(name="pack_rmat20_t4", op="pack", graph="rmat", scale=20, T=4),
    ]


def log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["full", "full", "bits", "count", "bfs", "multi", "spmm", "spmm", "train", "newgraph", "pack"])
    case = dict(op=op, T=rng.choice([4, 8, 16, 32]))
    heavy = op in ("spmm", "train", "newgraph", "pack")
    kind = rng.choice(["rmat", "er", "rect"] if op in ("full", "count", "spmm", "newgraph", "pack") else ["rmat", "er"])
    case["graph"] = kind
    if kind == "rmat":
        case["scale"] = rng.randint(12, 18 if heavy else 20)
    else:
        # at T = 32 a tile takes 132 bytes, so fewer vertices make the same matrix
        case["n"] = int(log_between(rng, 3000, 300000 if heavy or case["T"] == 32 else 1000000))
        case["degree"] = round(rng.uniform(4, 32), 1)
        if kind == "rect":
            case["ncols"] = int(case["n"] * log_between(rng, 0.3, 3))
    if op in ("bits", "count"):
        case["density"] = round(log_between(rng, 0.001, 0.5), 4)
    if op == "bits":
        case["masked"] = rng.random() < 0.5
    if op == "count":
        case["as_float"] = rng.random() < 0.5
    if op == "bfs":
        case["levels"] = rng.randint(3, 8)
    if op in ("bits", "bfs"):
        case["direction"] = rng.choice(["pull", "auto"])
    if op == "multi":
        case["word_bits"] = rng.choice([32, 64])
    if heavy and op != "pack":
        # feature widths: powers of two as often as any other
        case["k"] = rng.choice([16, 32, 64, 128]) if rng.random() < 0.5 else int(log_between(rng, 3, 160))
        case["fp64"] = op == "spmm" and rng.random() < 0.15
    return case
