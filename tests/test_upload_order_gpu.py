"""Tables that batch creation and admission write are read on streams that do
not wait for the legacy stream: a batch run on a non-blocking stream right
after its creation, and plans admitted into slots of a running server, give
each matrix's own multiply bit for bit."""
import ctypes as C

import numpy as np
import pytest

from taichi_b200 import matgen

pytestmark = pytest.mark.gpu


def make(tc, dev, n, seed):
    """Plans of n matrices of different sizes, x, and y of each plan alone."""
    import torch
    rng = np.random.default_rng(seed)
    plans, xs, want = [], [], []
    for i in range(n):
        M, N, rp, col = matgen.segments(600 + 137 * i, [(0, 600 + 137 * i, 0, 3, 0.9)], noise=400, seed=seed + i)
        plans.append(tc.Plan.from_csr(M, N, rp, col))
        xs.append(torch.from_numpy(rng.uniform(-1, 1, N).astype(np.float32)).to(dev))
        want.append(torch.empty(M, device=dev))
        plans[-1].spmv(xs[-1], want[-1])
    torch.cuda.synchronize()
    return plans, xs, want


@pytest.mark.parametrize("graph", [False, True])
def test_batch_run_at_once(tc, dev, graph):
    import torch
    plans, xs, want = make(tc, dev, 12, 3)
    side = torch.cuda.Stream()                       # non-blocking
    for turn in range(20):                           # tables of other sizes and contents in reused memory
        n = 1 + (7 * turn) % len(plans)
        order = np.random.default_rng(turn).permutation(len(plans))[:n]
        ys = [torch.full_like(want[i], float("nan")) for i in order]
        torch.cuda.synchronize()
        arr, b = C.c_void_p * n, C.c_void_p()
        tc.check(tc.lib().tc_batch_create(n, arr(*[plans[i].handle.value for i in order]),
                                          arr(*[xs[i].data_ptr() for i in order]),
                                          arr(*[y.data_ptr() for y in ys]), C.byref(b)))
        run = tc.lib().tc_batch_graph_launch if graph else tc.lib().tc_batch_run
        tc.check(run(b, C.c_void_p(side.cuda_stream)))
        side.synchronize()
        tc.check(tc.lib().tc_batch_destroy(b))
        for i, y in zip(order, ys):
            assert torch.equal(y, want[i])


def test_admit_while_serving(tc, dev):
    import torch
    plans, xs, want = make(tc, dev, 8, 40)
    srv = tc.Server(contexts=2, max_batch=8, max_inflight=2, arena_bytes=1 << 20)
    ids = [srv.admit(plans[0]), srv.admit(plans[1])]
    srv.start(device_vectors=True)
    for turn in range(40):                           # slot 0 changes hands, slot 1 stays
        i = turn % len(plans)
        srv.evict(ids[0])
        ids[0] = srv.admit(plans[i])
        ys = [torch.full_like(want[i], float("nan")), torch.full_like(want[1], float("nan"))]
        torch.cuda.synchronize()
        tickets = [srv.submit(ids[0], xs[i], ys[0]), srv.submit(ids[1], xs[1], ys[1])]
        for t in tickets:
            srv.wait(t, 30.0)
        assert torch.equal(ys[0], want[i]) and torch.equal(ys[1], want[1])
    srv.stop()
    srv.close()
