"""The double-precision multiply's row layouts (1, 4 and 8 lanes a row, tiles
with rows for a warp or a CTA) at their edges: integer x, where every partial
sum is exact, against the FP64 oracle, multiplied in a chain under
programmatic dependent launch."""
import numpy as np
import pytest

import oracle
from tests.test_mixed_tiles_gpu import matrix as mixed
from tests.test_spmm_layouts_gpu import csr_of, matrix as layouts

pytestmark = pytest.mark.gpu


def matrix(name):
    rng = np.random.default_rng(11)
    if name.startswith("rows"):                      # lanes 1, 4, 8 by the mean row length; ragged row counts
        mean, M = map(int, name[4:].split("x"))
        lens = np.clip(rng.poisson(mean, M), 0, 128)
        lens[M // 2] = 128
        return csr_of(lens, M + 200, mean)
    return mixed(name) if name in ("edges", "sparse", "powerlaw", "hybrid") else layouts(name)


@pytest.mark.parametrize("name", ["rows1x1", "rows3x257", "rows7x1023", "rows12x63", "rows12x65", "rows12x1000",
                                  "rows20x31", "rows20x33", "rows40x999", "edges", "sparse", "powerlaw", "hybrid",
                                  "hybrid1", "hybrid3", "hybrid13", "empty_tail"])
def test_layouts(tc, dev, name):
    import torch
    M, N, rp, col = matrix(name)
    plan = tc.Plan.from_csr(M, N, rp, col)
    x = np.random.default_rng(1).integers(-8, 9, N).astype(np.float64)
    xd = torch.from_numpy(x).to(dev)
    steps = 3 if M == N else 1                       # v <- A v: integers below 2^53
    want = x
    for _ in range(steps):
        y = torch.full((M,), float("nan"), dtype=torch.float64, device=dev)
        plan.spmv_f64(xd, y)
        xd = y
        want = oracle.spmv_csr_f64(M, rp, col, want)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(y.cpu().numpy(), want)


@pytest.mark.parametrize("more", [-1, 0, 1, 127])
@pytest.mark.parametrize("mean", [9, 17, 18, 29])
@pytest.mark.parametrize("wave", [512, 1024])
def test_lanes(tc, dev, wave, mean, more):
    """Rows about the lengths and the numbers from which two, four or eight
    lanes share one (8 CTAs of 128 and of 64 rows per multiprocessor)."""
    import torch
    M = wave * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(mean)
    lens = np.full(M, mean)
    lens[[1, M - 1]] = [mean - 9, mean + 9]          # the mean as it is, not every row the same
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    col = rng.integers(0, M, rp[-1]).astype(np.int32)
    plan = tc.Plan.from_csr(M, M, rp, col, partition=False)
    x = rng.integers(-8, 9, M)
    y = torch.full((M,), float("nan"), dtype=torch.float64, device=dev)
    plan.spmv_f64(torch.from_numpy(x.astype(np.float64)).to(dev), y)
    torch.cuda.synchronize()
    sums = np.concatenate([[0], np.cumsum(x[col])])
    np.testing.assert_array_equal(y.cpu().numpy().astype(np.int64), sums[rp[1:]] - sums[rp[:-1]])


def test_no_columns(tc, dev):
    import torch
    plan = tc.Plan.from_csr(40, 0, np.zeros(41, np.int32), np.zeros(0, np.int32), partition=False)
    y = torch.ones(40, dtype=torch.float64, device=dev)
    plan.spmv_f64(y, y)
    torch.cuda.synchronize()
    assert not y.any()
