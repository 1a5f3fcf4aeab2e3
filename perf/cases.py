"""Performance cases of taichi_b200: what its users run, through its public
entry points (Plan, tc_batch_*, Server).

    listed()            the cases that are tracked
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call (plans, vectors)
    run(state)          one pass
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   what run() returns, from torch in 64 bits

A case names an operation (`op`), a matrix family (`family`) and their sizes:

    spmv      y = A x, one tc_spmv per pass
    iterate   v <- A v, `steps` times, as one replay of a captured CUDA graph
    spmv64    y = A x with double-precision vectors (tc_spmv_f64)
    spmm      Y = A X for `rhs` right-hand sides (tc_spmm)
    batch     `count` resident matrices of uneven size, one graph launch
    build     device CSR -> plan (partition and format build), first multiply
    serve     `requests` requests over `count` resident matrices, all waiting
              when the pass starts (tc_server_run, device vectors)

Families, all generated on the GPU from the seed:

    rmat      R-MAT graph of 2^scale rows, quadrants (a, b, b, 1 - a - 2b),
              `ef` edges per row drawn, duplicates removed; self-loops kept
              only with loops = True.  a = 0.499, b = 0.001 gives graphs whose
              entries gather near the diagonal (under one per row); a = 0.57,
              b = 0.19 the power-law graphs of the graph benchmarks
    mesh      9-point stencil on a grid x grid mesh, 2 % of the rows' contents
              exchanged among themselves
    banded    dense diagonals -k..+k plus `extra` uniform random columns a row
    segment   dense diagonals -k..+k, 95 % of each kept, plus one random
              entry per ten rows (dense diagonals with holes and left-overs)

Vectors are uniform in [-1, 1].
"""
import ctypes
import math

import torch

import taichi_b200 as tc

DEV = "cuda"
NEAR = {"ef": 16, "a": 0.499, "b": 0.001}
POWER = {"ef": 16, "a": 0.57, "b": 0.19}


def listed():
    return [
        # the small matrix whose diagonals the partition leaves in the CSR
        # (65,536 rows of 18 entries): a launch and one wave of tiles
        dict(name="spmv_small", op="spmv", family="banded", n=65536, k=4, extra=10),
        # an iterative method on the R-MAT graph of the headline benchmark,
        # its multiplies captured once and replayed
        dict(name="iterate_rmat20", op="iterate", family="rmat", scale=20, loops=False, steps=8, **NEAR),
        # a large structured-grid operator with irregular rows: the hybrid
        # format at full size
        dict(name="spmv_mesh2048", op="spmv", family="mesh", grid=2048),
        # the largest kind of matrix a served pool holds: wide rows that the
        # partition leaves plain, an odd number of them
        dict(name="spmv_banded", op="spmv", family="banded", n=2279375, k=12, extra=7),
        # a web- or social-network-like graph: empty rows beside rows of
        # tens of thousands of entries
        dict(name="spmv_powerlaw", op="spmv", family="rmat", scale=20, loops=False, **POWER),
        # a solver that keeps its vectors in double precision, ragged grid
        dict(name="spmv64_mesh", op="spmv64", family="mesh", grid=1531),
        # many right-hand sides on a large graph (embedding propagation)
        dict(name="spmm_rmat22_k64", op="spmm", family="rmat", scale=22, loops=False, rhs=64, **NEAR),
        # a block of a few vectors on a grid operator (block eigensolvers)
        dict(name="spmm_mesh_k8", op="spmm", family="mesh", grid=1200, rhs=8),
        # many independent systems of uneven size in one launch
        dict(name="batch256", op="batch", count=256),
        # a new matrix: partition, format build and the first multiply,
        # once with dense diagonals and holes, once on the large graph whose
        # self-loops make one dense diagonal
        dict(name="build_mesh2048", op="build", family="mesh", grid=2048),
        dict(name="build_rmat20_loops", op="build", family="rmat", scale=20, loops=True, **NEAR),
        # a server with a backlog: requests over a pool of resident matrices
        dict(name="serve_pool", op="serve", count=16, requests=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, entries):
    """A matrix family and size of at most about `entries` entries."""
    family = rng.choice(["rmat", "power", "mesh", "banded", "segment"])
    if family == "rmat":
        top = 22 if entries >= 2.5e6 else 21 if entries >= 1.7e6 else 19
        return dict(family="rmat", scale=rng.randint(12, top), loops=rng.random() < 0.3, **NEAR)
    if family == "power":
        return dict(family="rmat", scale=rng.randint(11, min(20, int(math.log2(entries / 16)))), loops=False, **POWER)
    if family == "mesh":
        return dict(family="mesh", grid=_log(rng, 64, math.sqrt(min(entries, 3.77e7) / 9)))
    k = rng.randint(1, 12)
    if family == "banded":
        extra = rng.randint(2, 10)
        return dict(family="banded", n=_log(rng, 4000, min(2.2e6, entries / (2 * k + 1 + extra))), k=k, extra=extra)
    return dict(family="segment", n=_log(rng, 20000, max(30000, min(2.2e6, entries / (2 * k + 1)))), k=k)


def draw(rng):
    op = rng.choice(["spmv", "spmv", "spmv", "iterate", "spmv64", "spmm", "spmm", "batch", "build", "serve"])
    if op == "batch":
        return dict(op=op, count=_log(rng, 16, 255))
    if op == "serve":
        return dict(op=op, count=rng.randint(4, 16), requests=_log(rng, 8, 255))
    if op == "spmm":
        rhs = _log(rng, 1, 64)
        return dict(op=op, rhs=rhs, **_matrix(rng, min(1.2e7, 3e8 / rhs)))
    c = dict(op=op, **_matrix(rng, 3e7 if op == "spmv" else 1.5e7))
    if op == "iterate":
        c["steps"] = rng.randint(2, 8)
    return c


# ---------------------------------------------------------------- matrices
def _gen(seed):
    return torch.Generator(DEV).manual_seed(seed)


def _csr(M, N, keys):
    """CSR of sorted unique keys row * N + column."""
    rows = torch.div(keys, N, rounding_mode="floor")
    rowptr = torch.zeros(M + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(rows, minlength=M), 0, out=rowptr[1:])
    return M, rowptr.int(), (keys - rows * N).int()


def _rmat(scale, ef, a, b, loops, g):
    n = 1 << scale
    r = torch.zeros(ef * n, dtype=torch.int64, device=DEV)
    c = torch.zeros_like(r)
    for _ in range(scale):
        u = torch.rand(ef * n, device=DEV, generator=g)
        low = u >= a + b
        r = r * 2 + low
        c = c * 2 + (((u >= a) & ~low) | (u >= a + 2 * b))
    keys = r * n + c
    if not loops:
        keys = keys[r != c]
    return _csr(n, n, torch.unique(keys))


def _mesh(grid, g):
    n = grid * grid
    i = torch.arange(n, device=DEV)
    moved = torch.randperm(n, device=DEV, generator=g)[: n // 50]
    i[moved.sort().values] = moved
    y, x = torch.div(i, grid, rounding_mode="floor"), i % grid
    d = torch.tensor([-1, 0, 1], device=DEV)
    dy, dx = d.repeat_interleave(3), d.repeat(3)
    yy, xx = y[:, None] + dy, x[:, None] + dx
    ok = (yy >= 0) & (yy < grid) & (xx >= 0) & (xx < grid)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(ok.sum(1), 0, out=rowptr[1:])
    return n, rowptr.int(), (yy * grid + xx)[ok].int()


def _banded(n, k, extra, keep, g):
    r = torch.arange(n, device=DEV)
    c = r[:, None] + torch.arange(-k, k + 1, device=DEV)
    ok = (c >= 0) & (c < n)
    if keep < 1:
        ok &= torch.rand(c.shape, device=DEV, generator=g) < keep
    keys = [(r[:, None] * n + c)[ok]]
    more = int(extra * n)
    rows = r.repeat_interleave(extra) if extra >= 1 else torch.randint(n, (more,), device=DEV, generator=g)
    keys.append(rows * n + torch.randint(n, (more,), device=DEV, generator=g))
    return _csr(n, n, torch.unique(torch.cat(keys)))


def _matrix_of(c, g):
    """(M, rowptr, col) of the case's matrix, int32 CSR on the GPU."""
    if c["family"] == "rmat":
        return _rmat(c["scale"], c["ef"], c["a"], c["b"], c["loops"], g)
    if c["family"] == "mesh":
        return _mesh(c["grid"], g)
    if c["family"] == "banded":
        return _banded(c["n"], c["k"], c["extra"], 1.0, g)
    return _banded(c["n"], c["k"], 0.1, 0.95, g)


def _pool(c, g):
    """The matrices of a batch or of a served pool: even ones R-MAT, odd ones
    banded plus random columns, sizes spread over their logarithm (the case's
    own sizes; the entries follow the seed)."""
    pick = torch.rand(3 * c["count"], generator=torch.Generator().manual_seed(c["count"])).tolist()
    out = []
    for i in range(c["count"]):
        u, v, w = pick[3 * i: 3 * i + 3]
        if c["op"] == "batch":
            n = int(1000 * 200 ** u)
            out.append(_rmat(max(10, round(math.log2(n))), 8, 0.499, 0.001, False, g) if i % 2 == 0
                       else _banded(n, 1 + int(16 * v), 4, 1.0, g))
        elif i % 2 == 0:
            out.append(_rmat(14 + int(8 * u), 16, 0.499, 0.001, False, g))
        else:
            out.append(_banded(int(1e4 * 100 ** u), 1 + int(16 * v), 2 + int(11 * w), 1.0, g))
    return out


def _requests(c):
    """The matrix of each request: Zipf(1.1) over the pool in a shuffled order."""
    g = torch.Generator().manual_seed(c["requests"])
    weight = torch.arange(1, c["count"] + 1, dtype=torch.float64) ** -1.1
    order = torch.randperm(c["count"], generator=g)
    return order[torch.multinomial(weight, c["requests"], True, generator=g)].tolist()


def _uniform(shape, g, dtype=torch.float32):
    return torch.rand(shape, device=DEV, generator=g, dtype=dtype) * 2 - 1


def _offsets(sizes):
    """Starts of 256-byte aligned float vectors packed in one buffer."""
    at = [0]
    for n in sizes:
        at.append(at[-1] + (n + 63) // 64 * 64)
    return at


def _inputs(c, seed):
    """Matrices and vectors of the case: (matrices, x); x packed for a pool."""
    g = _gen(seed)
    if c["op"] in ("batch", "serve"):
        pool = _pool(c, g)
        owner = range(len(pool)) if c["op"] == "batch" else _requests(c)
        at = _offsets([pool[i][0] for i in owner])
        return pool, list(owner), at, _uniform(at[-1], g)
    m = _matrix_of(c, g)
    if c["op"] == "spmm":
        return [m], None, None, _uniform((m[0], c["rhs"]), g)
    return [m], None, None, _uniform(m[0], g, torch.float64 if c["op"] == "spmv64" else torch.float32)


# -------------------------------------------------------------------- state
class Batch:
    """tc_batch over plans, x and y vectors."""

    def __init__(self, plans, xs, ys):
        n = len(plans)
        arr = ctypes.c_void_p * n
        self.plans = plans
        self.handle = ctypes.c_void_p()
        tc.check(tc.lib().tc_batch_create(n, arr(*[p.handle for p in plans]), arr(*[x.data_ptr() for x in xs]),
                                          arr(*[y.data_ptr() for y in ys]), ctypes.byref(self.handle)))

    def launch(self):
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        tc.check(tc.lib().tc_batch_graph_launch(self.handle, stream))

    def __del__(self):
        tc.lib().tc_batch_destroy(self.handle)


def _plan(m):
    return tc.Plan.from_csr(m[0], m[0], m[1], m[2], on_device=True)


def prepare(case, seed):
    pool, owner, at, x = _inputs(case, seed)
    s = dict(op=case["op"], x=x)
    if case["op"] == "build":
        s.update(matrix=pool[0], plan=None, y=torch.empty_like(x))
        return s
    plans = [_plan(m) for m in pool]
    s["y"] = torch.zeros_like(x)
    if case["op"] in ("batch", "serve"):
        xs = [x[a: a + pool[i][0]] for a, i in zip(at, owner)]
        ys = [s["y"][a: a + pool[i][0]] for a, i in zip(at, owner)]
        if case["op"] == "batch":
            s["batch"] = Batch(plans, xs, ys)
        else:
            s["server"] = tc.Server()
            ids = [s["server"].admit(p) for p in plans]
            s.update(arrival=[0.0] * len(owner), matrix=[ids[i] for i in owner], xs=xs, ys=ys)
        return s
    s["plan"] = plans[0]
    if case["op"] == "iterate":
        v = [x, s["y"], torch.zeros_like(x)]
        plans[0].spmv(x, s["y"])
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            for i in range(case["steps"]):
                plans[0].spmv(v[0] if i == 0 else v[1 + (i - 1) % 2], v[1 + i % 2], stream=torch.cuda.current_stream())
        s.update(y=v[1 + (case["steps"] - 1) % 2], vectors=v)
    return s


def run(s):
    op = s["op"]
    if op == "spmv":
        s["plan"].spmv(s["x"], s["y"])
    elif op == "iterate":
        s["graph"].replay()
    elif op == "spmv64":
        s["plan"].spmv_f64(s["x"], s["y"])
    elif op == "spmm":
        s["plan"].spmm(s["x"], s["y"])
    elif op == "batch":
        s["batch"].launch()
    elif op == "serve":
        s["server"].run(s["arrival"], s["matrix"], s["xs"], s["ys"], mode=tc.SERVE_DEVICE_VECTORS)
    else:
        # a program that follows a changing matrix: the new plan replaces the old
        s["plan"] = _plan(s["matrix"])
        s["plan"].spmv(s["x"], s["y"])
        i = s["plan"].info()
        return dict(y=s["y"], format=[i[k] for k in ("dia_shapes", "num_negs", "dense_nnz", "zero_elements",
                                                     "sparse_nnz", "row_start", "row_stop", "nnz_csr")])
    return s["y"]


# --------------------------------------------------------------- the bounds
def work(case):
    """Formatted matrix, x and y each moved once per multiply (a vector value
    counts 8 bytes in spmv64); a build reads the input CSR and writes the
    format besides.  Two operations per entry and right-hand side."""
    pool, owner, _, _ = _inputs(case, 0)
    nbytes = flops = 0
    infos = []
    for m in pool:
        p = _plan(m)
        infos.append(p.info())
        p.close()
    for i in owner if owner is not None else [0]:
        n, rowptr, col = pool[i]
        fmt = infos[i]["spmv_bytes"] - 8 * n
        k, size = (case["rhs"], 4) if case["op"] == "spmm" else (1, 8 if case["op"] == "spmv64" else 4)
        nbytes += fmt + 2 * size * k * n
        flops += 2 * k * col.numel()
        if case["op"] == "build":
            nbytes += 4 * (rowptr.numel() + col.numel()) + fmt
    return {"bytes": nbytes * case.get("steps", 1), "flops": flops * case.get("steps", 1)}


def exact(case, seed):
    pool, owner, at, x = _inputs(case, seed)
    x = x.double()

    def multiply(m, v):
        n, rowptr, col = m
        rows = torch.repeat_interleave(torch.arange(n, device=DEV), rowptr.diff().long())
        y = torch.zeros_like(v)
        if v.dim() == 1:
            return y.index_add_(0, rows, v[col.long()])
        for c0 in range(0, v.shape[1], 8):        # a few columns at a time: the terms take memory
            part = torch.zeros_like(v[:, c0: c0 + 8]).contiguous()
            y[:, c0: c0 + 8] = part.index_add_(0, rows, v[:, c0: c0 + 8][col.long()])
        return y

    if owner is not None:
        y = torch.zeros_like(x)
        for a, i in zip(at, owner):
            n = pool[i][0]
            y[a: a + n] = multiply(pool[i], x[a: a + n])
        return y
    for _ in range(case.get("steps", 1)):
        x = multiply(pool[0], x)
    return dict(y=x, format=None) if case["op"] == "build" else x
