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


def test_no_columns(tc, dev):
    import torch
    plan = tc.Plan.from_csr(40, 0, np.zeros(41, np.int32), np.zeros(0, np.int32), partition=False)
    y = torch.ones(40, dtype=torch.float64, device=dev)
    plan.spmv_f64(y, y)
    torch.cuda.synchronize()
    assert not y.any()
