"""Stream plans of just as many tiles as one wave of CTAs holds at 5 and at 6
CTAs per multiprocessor, and one more (at 148 multiprocessors), plain and with
dense diagonals: integer x against numpy, the batched launch bit-identical."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [740, 741, 888, 889])
@pytest.mark.parametrize("diags", [0, 2])
def test_wave_edges(tc, dev, tiles, diags):
    import torch
    M, per = 256 * tiles, 12
    rng = np.random.default_rng(tiles + diags)
    col = rng.integers(0, M, M * per).astype(np.int32)
    sign = np.where(rng.random(M * per) < 0.8, 1, -1) if diags else np.ones(M * per, np.int64)
    words = (col << 1) | (sign > 0) if diags else col
    f = dict(dia_shapes=int(diags > 0), num_negs=diags, dense_nnz=int(diags > 0), zero_elements=0,
             sparse_nnz=M * per, row_start=0, row_stop=M if diags else 0, xStart=[0], yStart=[0], xStop=[M],
             nDiasPtr=[0, diags], neg_offsets=[0, 1][:diags] or [0],
             csrRow=np.arange(0, M * per + 1, per, dtype=np.int32), csrCol=words.astype(np.int32))
    plan = tc.Plan.from_format(M, M, f)
    assert plan.info()["ntiles"] == tiles and plan.info()["kernel"] == 4
    x = rng.integers(-8, 9, M).astype(np.float32)
    want = (x[col] * sign).reshape(M, per).sum(1).astype(np.float64)
    if diags:
        want += x
        want[:-1] += x[1:]
    xd, y, yb = torch.from_numpy(x).to(dev), torch.empty(M, device=dev), torch.empty(M, device=dev)
    plan.spmv(xd, y)
    b, one = C.c_void_p(), C.c_void_p * 1
    tc.check(tc.lib().tc_batch_create(1, one(plan.handle.value), one(xd.data_ptr()), one(yb.data_ptr()), C.byref(b)))
    tc.check(tc.lib().tc_batch_run(b, None))
    torch.cuda.synchronize()
    tc.check(tc.lib().tc_batch_destroy(b))
    np.testing.assert_array_equal(y.cpu().numpy().astype(np.float64), want)
    assert torch.equal(y, yb)
