"""The memory a build leaves with the library: at most 256 MB beyond the plan
itself when the call returns, whatever scratch the build took, without a wait
of the program's own; builds from several threads and streams at once share
the pool and give the plans that they give one after the other."""
import threading

import numpy as np
import pytest

from taichi_b200 import matgen

pytestmark = pytest.mark.gpu
MB = 1 << 20


def big(tc):
    """A matrix of 100 M entries: 400 MB of columns."""
    M, per = 1_000_000, 100
    col = (np.arange(per, dtype=np.int32) * 9973)[None, :] + np.arange(M, dtype=np.int32)[:, None]
    return M, np.arange(0, M * per + 1, per, dtype=np.int32), np.ascontiguousarray(col % M).reshape(-1)


@pytest.mark.parametrize("flags", ["partition", "plain"])
def test_build_from_host_arrays(tc, dev, flags):
    import torch
    M, rp, col = big(tc)
    small = matgen.segments(2000, [(0, 2000, 0, 3, 0.9)], noise=500, seed=1)
    first = tc.Plan.from_csr(*small)                    # the pool exists, and a plan keeps it from being trimmed
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    prm = tc.params(flags=1) if flags == "plain" else None
    plan = tc.Plan.from_csr(M, M, rp, col, prm=prm)
    held = before - torch.cuda.mem_get_info()[0] - plan.info()["device_bytes"]
    print("held beyond the plan: %.0f MB" % (held / MB))
    # 256 MB and the allocators' granularity (2 MB pages, 32 MB pool blocks)
    assert held <= (256 + 40) * MB
    plan.close()
    first.close()


def test_builds_from_threads(tc, dev):
    import torch
    mats = [matgen.segments(3000 + 611 * i, [(0, 3000, 0, 4, 0.9), (200, 2900, 40 * i, 1, 0.95)], noise=2000, seed=i)
            for i in range(6)]
    want = [tc.Plan.from_csr(*m).export() for m in mats]
    fails = []

    def work(t):
        try:
            s = torch.cuda.Stream()
            for turn in range(12):
                i = (t + turn) % len(mats)
                M, N, rp, col = mats[i]
                if turn % 2:
                    with torch.cuda.stream(s):
                        a, b = torch.from_numpy(rp).to(dev), torch.from_numpy(col).to(dev)
                    s.synchronize()
                    plan = tc.Plan.from_csr(M, N, a, b, on_device=True, stream=s)
                else:
                    plan = tc.Plan.from_csr(M, N, rp, col, stream=s)
                got = plan.export()
                for k in ("csrRow", "csrCol", "neg_offsets", "xStart"):
                    np.testing.assert_array_equal(got[k], want[i][k], err_msg="%d %s" % (i, k))
                x = torch.ones(N, device=dev)
                y = torch.empty(M, device=dev)
                torch.cuda.synchronize()
                plan.spmv(x, y, stream=s)
                s.synchronize()
                np.testing.assert_array_equal(y.cpu().numpy(), np.diff(rp).astype(np.float32))
                plan.close()
        except Exception as e:                          # noqa: BLE001 -- reported by the main thread
            fails.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fails, fails[0]
