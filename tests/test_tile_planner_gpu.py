"""The tile planner against a restatement of its rules in Python: how many
tiles, long tiles and lane tiles a plan of each tile mode has, for short rows,
rows of every length, long rows, rows past the word limits, and matrices of
more than one strip of rows; and y against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STRIP, SPAN, BLOCK = 16384, 2048, 256


def lanes_for(mean, most):
    if mean <= 16:
        return 1
    n = 1
    while n < most and 8.0 * n < mean:
        n *= 2
    return n


def plan(lens, sms, mode=2, tile_rows=1024, tile_nnz=2048, strided=False, no_direct=False):
    """(tiles, long tiles, lane tiles) of a plan that is not wide."""
    nnz, tiles, longs, vector = int(lens.sum()), 0, 0, 0
    spread = min(4096, max(512, nnz // (4 * sms)))
    long_len = max(1, min(tile_nnz, 4096 if mode == 2 else 8192))
    cap_nnz = max(1, min(2 * tile_nnz, spread))
    for lo in range(0, len(lens), STRIP):
        part = lens[lo:lo + STRIP]
        rp = np.concatenate([[0], np.cumsum(part)])
        over = np.append(np.flatnonzero(part > long_len), len(part))
        mids = np.append(np.flatnonzero(part > 128), len(part))
        n, r = len(part), 0
        while r < n:
            if part[r] > long_len:
                tiles, longs, r = tiles + 1, longs + 1, r + 1
                continue
            stop = over[np.searchsorted(over, r)]
            if mode == 2:
                a4 = r % 4 == 0 and not strided
                end = min(n, r // SPAN * SPAN + SPAN) if lens.max() > 128 else n
                m = min(np.searchsorted(rp, rp[r] + cap_nnz, "right") - 1 - r, min(tile_rows, 1024 if a4 else 256), stop - r, end - r)
                m = max(int(m), 1)
                small = min(m, mids[np.searchsorted(mids, r)] - r)
                if small >= 2 * BLOCK:
                    m = small
                ent = rp[r + m] - rp[r]
                direct = a4 and small >= 2 * BLOCK and ent <= m and not no_direct
                four = not direct and a4 and small >= 2 * BLOCK and ent <= 2 * m
                if not direct:
                    m = min(m, 1024 if four else 256)
                if r + m < end:
                    cut = (r + m) // 256 * 256
                    m = cut - r if cut - r >= 256 else m - (r + m) % 4 if m > 4 else m
            else:
                m = min(min(tile_rows, 2048) if mode == 0 else 1024, stop - r)
                if mode == 1:
                    m = min(m, BLOCK // lanes_for((rp[r + m] - rp[r]) / m, 32) * 4, tile_rows)
                while m > 1 and rp[r + m] - rp[r] > 8192:
                    m = (m + 1) // 2
                if mode == 1:
                    vector += lanes_for((rp[r + m] - rp[r]) / m, 32) > 1
            tiles, r = tiles + 1, r + m
    return tiles, longs, vector


def row_lengths(kind, rng):
    if kind == "short":
        return rng.poisson(2.5, 40001)
    if kind == "even":
        return np.full(100003, 18)
    if kind == "edges":
        return np.tile([0, 1, 127, 128, 129, 0, 0, 2047, 2048, 2049, 3, 3, 4095, 4096, 4097, 8192, 8193, 5], 60)
    if kind == "sparse":                              # direct and four-row runs between long rows
        lens = rng.choice([0, 0, 0, 1, 2], 50000)
        lens[rng.choice(50000, 40, replace=False)] = rng.integers(100, 3000, 40)
        return lens
    if kind == "mixed":
        return np.where(rng.random(35000) < 0.02, rng.integers(129, 900, 35000), rng.poisson(6, 35000))
    return np.array([3])


@pytest.mark.parametrize("kind", ["short", "even", "edges", "sparse", "mixed", "one"])
@pytest.mark.parametrize("over", [{}, {"tile_nnz": 16}, {"tile_nnz": 3, "tile_rows": 5}, {"tile_rows": 300},
                                  {"flags": 0x8}, {"flags": 0x10}, {"tile_mode": 0}, {"tile_mode": 0, "tile_rows": 5000},
                                  {"tile_mode": 1}, {"tile_mode": 1, "tile_rows": 77}],
                         ids=lambda o: ",".join("%s=%s" % kv for kv in o.items()) or "default")
def test_tiles(tc, dev, kind, over):
    import torch
    rng = np.random.default_rng(5)
    lens = row_lengths(kind, rng).astype(np.int64)
    M = len(lens)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, M, rp[-1]).astype(np.int32)
    prm = tc.params(**dict(over, flags=over.get("flags", 0) | 0x1 | 0x20))      # plain CSR, never wide
    p = tc.Plan.from_csr(M, M, rp, col, prm=prm)
    i = p.info()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    want = plan(lens, sms, over.get("tile_mode", 2), over.get("tile_rows", 1024), over.get("tile_nnz", 2048),
                over.get("flags", 0) == 0x8, over.get("flags", 0) == 0x10)
    assert (i["ntiles"], i["ntiles_long"], i["ntiles_vector"]) == want
    x = rng.integers(-8, 9, M)
    y = torch.full((M,), float("nan"), device=dev)
    p.spmv(torch.from_numpy(x.astype(np.float32)).to(dev), y)
    sums = np.concatenate([[0], np.cumsum(x[col])])
    np.testing.assert_array_equal(y.cpu().numpy().astype(np.int64), sums[rp[1:]] - sums[rp[:-1]])
