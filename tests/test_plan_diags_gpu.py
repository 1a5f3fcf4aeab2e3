"""Hybrid plans whose diagonals come with the launch parameters, at the edges
of that: 1, 4, 5, 8, 9, 33, 64 and 65 offsets (the last from the shape
arrays), shapes that end inside the matrix, off the main diagonal, and cut by
the format's row range: FP32, FP64 and four right-hand sides against numpy
for integer x, batched launch bit-identical."""
import ctypes as C

import numpy as np
import pytest


pytestmark = pytest.mark.gpu


def hybrid(M, N, x0, x1, y0, offs, seed, cut=(0, 0)):
    """A format with one shape (rows [x0, x1), columns from y0) and a random
    remainder of holes and left-overs, and its dense meaning as a CSR."""
    rng = np.random.default_rng(seed)
    words, rp = [], np.zeros(M + 1, np.int32)
    for r in range(M):
        n = int(rng.integers(0, 4))
        words += ((rng.integers(0, N, n) << 1) | (rng.random(n) < 0.7)).tolist()
        rp[r + 1] = len(words)
    return dict(dia_shapes=1, num_negs=len(offs), dense_nnz=1, zero_elements=0, sparse_nnz=len(words),
                row_start=x0 + cut[0], row_stop=x1 - cut[1], xStart=[x0], yStart=[y0], xStop=[x1],
                nDiasPtr=[0, len(offs)], neg_offsets=offs, csrRow=rp, csrCol=np.array(words + [0], np.int32)[:len(words)])


def dense_multiply(f, M, x):
    y = np.zeros((M,) + x.shape[1:])
    rows = np.repeat(np.arange(M), np.diff(f["csrRow"]))
    w = f["csrCol"]
    np.add.at(y, rows, np.where(w & 1, 1.0, -1.0).reshape((-1,) + (1,) * (x.ndim - 1)) * x[w >> 1])
    x0, x1, y0 = f["xStart"][0], f["xStop"][0], f["yStart"][0]
    for off in f["neg_offsets"]:
        r = np.arange(x0, x1)
        r = r[(r - x0 + off >= 0) & (r - x0 + off < x1 - x0) & (r >= f["row_start"]) & (r < f["row_stop"])]
        y[r] += x[r - x0 + y0 + off]
    return y


@pytest.mark.parametrize("noffs", [1, 4, 5, 8, 9, 33, 64, 65])
@pytest.mark.parametrize("box", ["whole", "inside", "cut"])
def test_offsets(tc, dev, noffs, box):
    import torch
    M, N = 3001, 3300
    x0, x1, y0, cut = {"whole": (0, 3001, 0, (0, 0)), "inside": (700, 2500, 1100, (0, 0)),
                       "cut": (700, 2500, 300, (40, 77))}[box]
    offs = sorted(np.random.default_rng(noffs).choice(np.arange(-90, 90), noffs, replace=False).tolist())
    f = hybrid(M, N, x0, x1, y0, offs, noffs, cut)
    plan = tc.Plan.from_format(M, N, f)
    x = np.random.default_rng(2).integers(-8, 9, (N, 4)).astype(np.float64)
    want = dense_multiply(f, M, x)
    xd = torch.from_numpy(x[:, 0].astype(np.float32)).to(dev)
    y = torch.full((M,), float("nan"), device=dev)
    plan.spmv(xd, y)
    y64 = torch.full((M,), float("nan"), dtype=torch.float64, device=dev)
    plan.spmv_f64(torch.from_numpy(x[:, 0].copy()).to(dev), y64)
    Y = torch.full((M, 4), float("nan"), device=dev)
    plan.spmm(torch.from_numpy(x.astype(np.float32)).to(dev), Y)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(y.cpu().numpy().astype(np.float64), want[:, 0])
    np.testing.assert_array_equal(y64.cpu().numpy(), want[:, 0])
    np.testing.assert_array_equal(Y.cpu().numpy().astype(np.float64), want)
    xf = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, N).astype(np.float32)).to(dev)
    plan.spmv(xf, y)
    yb = torch.full((M,), float("nan"), device=dev)
    b, one = C.c_void_p(), C.c_void_p * 1
    tc.check(tc.lib().tc_batch_create(1, one(plan.handle.value), one(xf.data_ptr()), one(yb.data_ptr()), C.byref(b)))
    tc.check(tc.lib().tc_batch_run(b, None))
    torch.cuda.synchronize()
    tc.check(tc.lib().tc_batch_destroy(b))
    assert torch.equal(y, yb)


@pytest.mark.parametrize("tile_nnz", [16, 100, 128])
def test_rows_of_a_cta(tc, dev, tile_nnz):
    """Rows of more than tile_nnz words get a CTA each, which adds them in
    another order than one thread: the same y alone and in a batch."""
    import torch
    M, rng = 30000, np.random.default_rng(tile_nnz)
    lens = rng.poisson(1.5, M)
    lens[rng.choice(M, 300, replace=False)] = rng.integers(10, 129, 300)
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    words = ((rng.integers(0, M, rp[-1]) << 1) | (rng.random(rp[-1]) < 0.7)).astype(np.int32)
    f = dict(dia_shapes=1, num_negs=3, dense_nnz=1, zero_elements=0, sparse_nnz=len(words), row_start=0, row_stop=M,
             xStart=[0], yStart=[0], xStop=[M], nDiasPtr=[0, 3], neg_offsets=[-1, 0, 1], csrRow=rp, csrCol=words)
    plan = tc.Plan.from_format(M, M, f, prm=tc.params(tile_nnz=tile_nnz))
    x = rng.uniform(-1, 1, M).astype(np.float32)
    xd, y, yb = torch.from_numpy(x).to(dev), torch.empty(M, device=dev), torch.empty(M, device=dev)
    plan.spmv(xd, y)
    b, one = C.c_void_p(), C.c_void_p * 1
    tc.check(tc.lib().tc_batch_create(1, one(plan.handle.value), one(xd.data_ptr()), one(yb.data_ptr()), C.byref(b)))
    tc.check(tc.lib().tc_batch_run(b, None))
    torch.cuda.synchronize()
    tc.check(tc.lib().tc_batch_destroy(b))
    assert torch.equal(y, yb)
    want = dense_multiply(f, M, x.astype(np.float64))
    assert np.abs(y.cpu().numpy() - want).max() <= 131 * 131 * 2.0 ** -24   # 131 terms of at most 1, one rounding each


@pytest.mark.parametrize("M,mean,long,share,kernel", [
    (60001, 0.4, 8, 0.01, 5), (60001, 0.4, 9, 0.01, 5), (60001, 0.4, 128, 0.002, 5),    # up to a word a row
    (1212417, 0.3, 16, 0.001, 2), (1200001, 0.3, 16, 0.001, 5),                        # about four waves of rows
    (400001, 1.3, 32, 0.004, 5), (400001, 1.3, 33, 0.004, 2), (400001, 1.3, 20, 0.02, 2), (400001, 1.3, 128, 1e-5, 2),
    (400001, 1.3, 20, -0.08, 5)])                   # negative share: neighbours
def test_spread_rows(tc, dev, M, mean, long, share, kernel):
    """Hybrid plans of three diagonals on both sides of the rules that give
    them to the rows kernel (5) or to their tiles (2), which lie at 148
    multiprocessors: y against numpy, alone and in a batch."""
    import torch
    rng = np.random.default_rng(M + long)
    lens = np.minimum(rng.poisson(mean, M), 6)
    if share < 0:
        lens[M // 3:M // 3 - int(M * share)] = long
    else:
        lens[rng.choice(M, max(1, int(M * share)), replace=False)] = long
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    words = ((rng.integers(0, M, rp[-1]) << 1) | (rng.random(rp[-1]) < 0.7)).astype(np.int32)
    f = dict(dia_shapes=1, num_negs=3, dense_nnz=1, zero_elements=0, sparse_nnz=len(words), row_start=0, row_stop=M,
             xStart=[0], yStart=[0], xStop=[M], nDiasPtr=[0, 3], neg_offsets=[-1, 0, 2], csrRow=rp, csrCol=words)
    plan = tc.Plan.from_format(M, M, f)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert plan.info()["kernel"] == kernel
    x = rng.integers(-8, 9, M).astype(np.float64)
    xd, y, yb = torch.from_numpy(x.astype(np.float32)).to(dev), torch.empty(M, device=dev), torch.empty(M, device=dev)
    plan.spmv(xd, y)
    b, one = C.c_void_p(), C.c_void_p * 1
    tc.check(tc.lib().tc_batch_create(1, one(plan.handle.value), one(xd.data_ptr()), one(yb.data_ptr()), C.byref(b)))
    tc.check(tc.lib().tc_batch_run(b, None))
    torch.cuda.synchronize()
    tc.check(tc.lib().tc_batch_destroy(b))
    np.testing.assert_array_equal(y.cpu().numpy().astype(np.float64), dense_multiply(f, M, x))
    assert torch.equal(y, yb)


@pytest.mark.parametrize("diags", [0, 3])
@pytest.mark.parametrize("mean", [1, 6, 12, 30])
def test_no_prefetch(tc, dev, diags, mean):
    """TC_FLAG_NO_PREFETCH changes no result of any multiply."""
    import torch
    M, rng = 310001, np.random.default_rng(mean)
    lens = rng.poisson(mean, M)
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    col = rng.integers(0, M, rp[-1]).astype(np.int32)
    f = dict(dia_shapes=int(diags > 0), num_negs=diags, dense_nnz=diags, zero_elements=0, sparse_nnz=rp[-1], row_start=0,
             row_stop=M if diags else 0, xStart=[0], yStart=[0], xStop=[M], nDiasPtr=[0, diags], neg_offsets=[-1, 0, 1],
             csrRow=rp, csrCol=(col << 1) | 1 if diags else col)
    x = torch.rand(M, 16, device=dev)
    got = []
    for flags in (0, 0x2000):
        plan = tc.Plan.from_format(M, M, f, prm=tc.params(flags=flags))
        y, Y = torch.empty(M, device=dev), torch.empty(M, 16, device=dev)
        y64 = torch.empty(M, dtype=torch.float64, device=dev)
        plan.spmv(x[:, 0].contiguous(), y)
        plan.spmv_f64(x[:, 1].double(), y64)
        plan.spmm(x, Y)
        torch.cuda.synchronize()
        got.append((y, y64, Y))
    for a, b in zip(*got):
        assert torch.equal(a, b)
