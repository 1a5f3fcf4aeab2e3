"""SpMM over every lane layout (vector and single loads, groups of 1 to 32
lanes) and row class (runs of short rows, one row per group, rows left to a
warp, rows with a CTA of their own), at the edges of each: integer X, where
every partial sum is an exact float, against the FP64 oracle."""
import numpy as np
import pytest

import oracle
from taichi_b200 import matgen

pytestmark = pytest.mark.gpu


def csr_of(lens, N, seed):
    rng = np.random.default_rng(seed)
    rp = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    col = [np.sort(rng.choice(N, n, replace=False)) for n in lens]
    return len(lens), N, rp, np.concatenate(col + [np.zeros(0, np.int64)]).astype(np.int32)


def matrix(name):
    rng = np.random.default_rng(3)
    if name.startswith("short"):                    # run kernel: mean of at most two words a row
        M = int(name[5:])
        lens = rng.choice([0, 0, 1, 1, 2, 5], M)
        lens[-1] = min(64, 2 * M - int(lens[:-1].sum())) if M > 40 else 1
        return csr_of(lens, 300, M)
    if name == "even":                              # one row per group, more than 8 words on average
        return csr_of(rng.integers(5, 30, 777), 900, 1)
    if name == "few":                               # one row per group, at most 8
        return csr_of(np.append(rng.integers(3, 9, 640), 64), 900, 2)
    if name == "empty_tail":
        return csr_of([3] * 200 + [0] * 313, 50, 4)
    if name == "skewed":                            # warp rows, rows of a tile of their own
        lens = rng.integers(0, 12, 600)
        lens[[0, 1, 2, 50, 51, 300, 301, 302, 599]] = [5000, 2049, 2048, 65, 64, 1024, 1025, 129, 700]
        return csr_of(lens, 6000, 5)
    # dense diagonals with holes, some rows long: the hybrid format of each kernel
    M, N, rp, col = matgen.segments(9000, [(0, 9000, 0, {"hybrid1": 0, "hybrid3": 1, "hybrid13": 6}[name], 0.97)],
                                    noise=900, seed=6)
    if name != "hybrid13":
        return M, N, rp, col
    lens = np.diff(rp)
    rows = [col[rp[r]:rp[r + 1]] for r in range(M)]
    for r, n in ((17, 100), (18, 1500), (5000, 3000)):
        rows[r] = np.unique(np.append(rows[r], rng.choice(N, n, replace=False))).astype(np.int32)
        lens[r] = len(rows[r])
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    return M, N, rp, np.concatenate(rows)


# (k, extra columns of ldx and ldy, floats off 16-byte alignment)
LAYOUTS = [(1, 0, 0), (2, 0, 0), (3, 0, 0), (4, 0, 0), (4, 4, 2), (6, 0, 0), (8, 0, 0), (8, 1, 0), (12, 4, 0),
           (13, 0, 1), (16, 0, 0), (24, 0, 0), (31, 0, 0), (33, 0, 0), (40, 0, 0), (62, 0, 0), (63, 2, 0),
           (64, 0, 0), (64, 0, 1), (64, 0, 2)]
NAMES = ["short1", "short31", "short33", "short255", "short257", "short1000", "even", "few", "empty_tail", "skewed",
         "hybrid1", "hybrid3", "hybrid13"]


@pytest.mark.parametrize("name", NAMES)
def test_layouts(tc, dev, name):
    import torch
    M, N, rp, col = matrix(name)
    plan = tc.Plan.from_csr(M, N, rp, col)
    assert (plan.info()["dia_shapes"] > 0) == name.startswith("hybrid")
    rng = np.random.default_rng(8)
    for k, pad, off in LAYOUTS:
        X = rng.integers(-8, 9, (N, k)).astype(np.float32)
        want = oracle.spmm_csr_f64(M, rp, col, X.astype(np.float64))
        ld = k + pad
        # the last row ends with the allocation's last float; padding and the
        # floats before the first row hold NaN and stay as they are
        xb = torch.full((off + (N - 1) * ld + k,), float("nan"), device=dev)
        yb = torch.full((off + (M - 1) * ld + k,), float("nan"), device=dev)
        torch.as_strided(xb, (N, k), (ld, 1), off).copy_(torch.from_numpy(X))
        plan.spmm(xb.data_ptr() + 4 * off, yb.data_ptr() + 4 * off, k=k, ldx=ld, ldy=ld)
        torch.cuda.synchronize()
        Y = torch.as_strided(yb, (M, k), (ld, 1), off)
        np.testing.assert_array_equal(Y.cpu().numpy().astype(np.float64), want, err_msg=str((k, pad, off)))
        Y.fill_(float("nan"))
        assert bool(torch.isnan(yb).all()), (k, pad, off)


@pytest.mark.parametrize("more", [-1, 0, 1, 31, 255])
def test_runs(tc, dev, more):
    """Short plain rows about the number from which they run as runs (two CTAs
    of 256 rows per multiprocessor)."""
    import torch
    M = 512 * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(M)
    lens = rng.choice([0, 0, 1, 1, 2, 5], M)
    lens[[0, 31, 32, M - 1]] = [64, 0, 64, 40]
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    col = rng.integers(0, 3000, rp[-1]).astype(np.int32)
    plan = tc.Plan.from_csr(M, 3000, rp, col, partition=False)
    for k in (5, 16, 29, 32, 64):
        X = rng.integers(-8, 9, (3000, k)).astype(np.float32)
        Y = torch.full((M, k), float("nan"), device=dev)
        plan.spmm(torch.from_numpy(X).to(dev), Y)
        torch.cuda.synchronize()
        sums = np.zeros((rp[-1] + 1, k))
        np.cumsum(X[col], axis=0, out=sums[1:], dtype=np.float64)
        np.testing.assert_array_equal(Y.cpu().numpy().astype(np.float64), sums[rp[1:]] - sums[rp[:-1]], err_msg=str(k))


@pytest.mark.parametrize("name", ["wide", "direct", "hybrid"])
def test_large_tiles(tc, dev, name):
    """Plans with rows of more than 64 words whose tiles hold hundreds of short
    rows, dealt out to several CTAs: row counts off every boundary."""
    import torch
    M, N = {"wide": 40003, "direct": 9001, "hybrid": 30011}[name], 3000 if name != "hybrid" else 30011
    rng = np.random.default_rng(M)
    lens = rng.choice([0, 0, 1, 1, 2], M)
    lens[[0, 1, M // 2, M - 1]] = [65, 128, 100, 70]
    if name == "direct":
        lens[[5000, 5001]] = [1500, 5000]
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    col = rng.integers(0, N, rp[-1]).astype(np.int32)
    sign = np.ones(rp[-1])
    if name == "hybrid":
        sign = np.where(rng.random(rp[-1]) < 0.7, 1.0, -1.0)
        f = dict(dia_shapes=1, num_negs=3, dense_nnz=1, zero_elements=0, sparse_nnz=rp[-1], row_start=0, row_stop=M,
                 xStart=[0], yStart=[0], xStop=[M], nDiasPtr=[0, 3], neg_offsets=[-2, 0, 1], csrRow=rp,
                 csrCol=(col << 1) | (sign > 0))
        plan = tc.Plan.from_format(M, N, f)
    else:
        plan = tc.Plan.from_csr(M, N, rp, col, partition=False)
    assert M // plan.info()["ntiles"] > 256 and (plan.info()["kernel"] == 3) == (name == "wide")
    for k in (1, 2, 5, 16, 29, 64):
        X = rng.integers(-8, 9, (N, k)).astype(np.float32)
        Y = torch.full((M, k), float("nan"), device=dev)
        plan.spmm(torch.from_numpy(X).to(dev), Y)
        torch.cuda.synchronize()
        sums = np.zeros((rp[-1] + 1, k))
        np.cumsum(X[col] * sign[:, None], axis=0, out=sums[1:])
        want = sums[rp[1:]] - sums[rp[:-1]]
        if name == "hybrid":
            want += X
            want[2:] += X[:-2]
            want[:-1] += X[1:]
        np.testing.assert_array_equal(Y.cpu().numpy().astype(np.float64), want, err_msg=str(k))


def test_non_finite_rows_stay_apart(tc, dev):
    """Slots past a row's words load X's row 0 and must not add it."""
    import torch
    for name in ("short1000", "few", "skewed", "hybrid3"):
        M, N, rp, col = matrix(name)
        plan = tc.Plan.from_csr(M, N, rp, col)
        X = np.ones((N, 8), np.float32)
        X[0] = np.inf
        Y = torch.zeros((M, 8), device=dev)
        plan.spmm(torch.from_numpy(X).to(dev), Y)
        torch.cuda.synchronize()
        touched = np.zeros(M, bool)
        touched[np.repeat(np.arange(M), np.diff(rp))[col == 0]] = True
        fmt = plan.export()                          # a hole in column 0 adds and subtracts it
        if fmt["dia_shapes"]:
            words, rows = fmt["csrCol"], np.repeat(np.arange(M), np.diff(fmt["csrRow"]))
            touched[rows[words >> 1 == 0]] = True
        np.testing.assert_array_equal(np.isfinite(Y.cpu().numpy()).all(1), ~touched, err_msg=name)


def test_no_columns(tc, dev):
    import torch
    plan = tc.Plan.from_csr(40, 0, np.zeros(41, np.int32), np.zeros(0, np.int32), partition=False)
    Y = torch.ones((40, 8), device=dev)
    plan.spmm(Y, Y, k=5, ldx=8, ldy=8)
    torch.cuda.synchronize()
    assert not Y[:, :5].any() and bool((Y[:, 5:] == 1).all())
