"""Mixed stream tiles (rows of more than 128 entries beside short ones in one
tile) at their edges: integer x against the FP64 oracle, and the same bits
from the batched and the served launch."""
import ctypes as C

import numpy as np
import pytest

import oracle
from taichi_b200 import matgen
from tests.test_spmm_layouts_gpu import csr_of

pytestmark = pytest.mark.gpu

EDGES = [127, 128, 129, 130, 0, 0, 1, 2047, 2048, 2049, 4095, 4096, 4097, 0, 5000, 131]


def matrix(name):
    rng = np.random.default_rng(7)
    if name == "edges":
        return csr_of(EDGES + [3] * 250 + EDGES, 6000, 1)
    if name == "eights":                             # usual row length 8: skewed slots
        lens = np.full(3000, 8)
        lens[rng.choice(3000, 120, replace=False)] = rng.integers(129, 900, 120)
        return csr_of(lens, 4000, 2)
    if name == "sparse":                             # direct and four-row runs between long rows
        lens = rng.choice([0, 0, 1, 1, 3], 9000)
        lens[[0, 1500, 4095, 4096, 8999]] = [200, 129, 3000, 300, 1000]
        return csr_of(lens, 9000, 3)
    if name == "powerlaw":
        M, N, rp, col = matgen.rmat(12, 16, 0.57, 0.19, 0.19, seed=4)
        return M, N, rp, col
    M, N, rp, col = matgen.segments(9000, [(0, 9000, 0, 1, 0.97)], noise=900, seed=6)    # hybrid
    rows = [col[rp[r]:rp[r + 1]] for r in range(M)]
    for r, n in ((0, 400), (17, 150), (5000, 3000), (8999, 129)):
        rows[r] = np.unique(np.append(rows[r], rng.choice(N, n, replace=False))).astype(np.int32)
    rp = np.zeros(M + 1, np.int32)
    np.cumsum([len(r) for r in rows], out=rp[1:])
    return M, N, rp, np.concatenate(rows)


@pytest.mark.parametrize("name", ["edges", "eights", "sparse", "powerlaw", "hybrid"])
def test_mixed_tiles(tc, dev, name):
    import torch
    M, N, rp, col = matrix(name)
    rng = np.random.default_rng(9)
    plan = tc.Plan.from_csr(M, N, rp, col)
    assert (plan.info()["dia_shapes"] > 0) == (name == "hybrid")
    for integer in (True, False):
        x = (rng.integers(-8, 9, N) if integer else rng.uniform(-1, 1, N)).astype(np.float32)
        xd = torch.from_numpy(x).to(dev)
        y = torch.full((M,), float("nan"), device=dev)
        plan.spmv(xd, y)
        torch.cuda.synchronize()
        if integer:
            np.testing.assert_array_equal(y.cpu().numpy().astype(np.float64),
                                          oracle.spmv_csr_f64(M, rp, col, x.astype(np.float64)))
        yb = torch.full((M,), float("nan"), device=dev)
        b, one = C.c_void_p(), C.c_void_p * 1
        tc.check(tc.lib().tc_batch_create(1, one(plan.handle.value), one(xd.data_ptr()), one(yb.data_ptr()), C.byref(b)))
        tc.check(tc.lib().tc_batch_run(b, None))
        torch.cuda.synchronize()
        tc.check(tc.lib().tc_batch_destroy(b))
        assert torch.equal(y, yb)
        server = tc.Server(solo_bytes=0)
        mid = server.admit(plan)
        ys = torch.full((M,), float("nan"), device=dev)
        server.run([0.0], [mid], [xd], [ys], mode=tc.SERVE_DEVICE_VECTORS)
        server.close()
        assert torch.equal(y, ys)


def test_served_in_large_launches(tc, dev):
    """Requests whose plans' own tiles come to more than a wave of CTAs (8 per
    multiprocessor) run the plans' tiles for large launches, also in one launch
    with smaller plans: each y as its plan alone gives it."""
    import torch
    rng = np.random.default_rng(4)
    names = ["edges", "eights", "sparse", "hybrid"]
    plans = [tc.Plan.from_csr(*matrix(n)) for n in names]
    M = 60000                                        # tiles of 512 words alone, of up to 4,096 in large launches
    plans.append(tc.Plan.from_csr(M, M, np.arange(0, 5 * M + 1, 5, dtype=np.int32),
                                  rng.integers(0, M, 5 * M).astype(np.int32), partition=False))
    sizes = [p.info() for p in plans]
    order = [4, 0, 4, 1, 4, 2, 4, 3] * 6
    wave = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    for at in range(len(order) - 4):                 # any five requests together are a large launch
        assert sum(sizes[i]["ntiles"] for i in order[at:at + 5]) > wave > sizes[4]["ntiles"]
    xs = [torch.from_numpy(rng.uniform(-1, 1, sizes[i]["N"]).astype(np.float32)).to(dev) for i in order]
    want = [torch.empty(sizes[i]["M"], device=dev) for i in order]
    for i, x, y in zip(order, xs, want):
        plans[i].spmv(x, y)
    server = tc.Server(solo_bytes=0, contexts=1, max_inflight=1)     # requests wait while a launch runs
    ids = [server.admit(p) for p in plans]
    ys = [torch.full_like(y, float("nan")) for y in want]
    torch.cuda.synchronize()
    stats, _ = server.run([0.0] * len(order), [ids[i] for i in order], xs, ys, mode=tc.SERVE_DEVICE_VECTORS)
    server.close()
    assert stats["mean_batch"] > 4
    for i, y, w in zip(order, ys, want):
        assert torch.equal(y, w), i
