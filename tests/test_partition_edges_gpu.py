"""The partitioner's run-based labelling, border walks and per-row hole bits
at the sizes where they can go wrong, bit for bit against the oracle: images
around word edges and too large for shared memory, opening lines longer than
a word, shapes of more than 32 dense diagonals, rows out of order and rows
with duplicate entries in one of several shapes."""
import ctypes as C

import numpy as np
import pytest

import oracle
from taichi_b200 import matgen

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 40), (40, 1), (5, 31), (33, 32), (32, 33), (17, 64), (65, 65), (97, 130), (300, 511),
         (1300, 1300)]


@pytest.mark.parametrize("H,W", SIZES)
def test_contours(tc, dev, H, W):
    rng = np.random.default_rng(H * 2000 + W)
    for density in (0.1, 0.45, 0.6, 0.9):
        img = (rng.random((H, W)) < density).astype(np.uint8)
        if density == 0.9 and min(H, W) > 20:
            img[2:-2, 2:-2] = 0                       # rings inside one another
            img[5:-5, 5:-5] = 1
            img[8:-8, 8:-8] = rng.random((H - 16, W - 16)) < 0.5
        want = oracle.find_contours(img)
        cap = H * W + 1
        lens, ends, n = np.zeros(cap, np.int32), np.zeros((cap, 4), np.int32), C.c_int()
        tc.check(tc.lib().tc_trace_contours(img.ctypes.data, H, W, lens.ctypes.data, ends.ctypes.data, cap,
                                            C.byref(n)))
        assert n.value == len(want)
        np.testing.assert_array_equal(lens[:n.value], [len(c) for c in want])
        if want:
            np.testing.assert_array_equal(ends[:n.value], [[*c[0], *c[len(c) // 2]] for c in want])


@pytest.mark.parametrize("height,open_len,eye", [(64, 1, 1), (64, 2, 4), (100, 31, 5), (333, 32, 5), (333, 33, 7),
                                                 (512, 40, 5), (1500, 30, 5)])
def test_thumbnail_stages(tc, dev, height, open_len, eye):
    M, N, rp, col = matgen.segments(4001, [(0, 2500, 0, 30, 0.97), (2000, 4001, -700, 60, 0.9), (500, 1500, 2000, 90, 1.0)],
                                    noise=6000, seed=height, n_cols=4100)
    over = dict(thumb_height=height, open_len=open_len, eye_size=eye, min_contour=20)
    mF, W, corners, stages = oracle.getsdf(M, N, rp, col, oracle.default_params(**over), stages=True)
    plan = tc.Plan.from_csr(M, N, rp, col, prm=tc.params(**over), keep_host=True)
    got_corners, got = plan.thumbnail(height)
    for k in range(5):
        np.testing.assert_array_equal(got[k] != 0, stages[k] != 0, err_msg="stage %d" % k)
    np.testing.assert_array_equal(got_corners, corners)


def rebuild(M, rows, col):
    rp = np.zeros(M + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=M), out=rp[1:])
    return rp, np.ascontiguousarray(col, np.int32)


@pytest.mark.parametrize("kind", ["sorted", "shuffled", "duplicates"])
@pytest.mark.parametrize("segs,many", [([(0, 4000, 0, 20, 0.93)], True),
                                       ([(0, 40000, 50000, 17, 0.97), (50000, 100000, -50000, 2, 0.95),
                                         (10000, 45000, 0, 0, 1.0)], True),
                                       ([(0, 9000, 40, 15, 1.0)], False)])
def test_hole_bits(tc, dev, kind, segs, many):
    n = max(s[1] for s in segs)
    M, N, rp, col = matgen.segments(n, segs, noise=min(n // 10, 1000), seed=8)
    rng = np.random.default_rng(2)
    rows = np.repeat(np.arange(M), np.diff(rp))
    if kind == "duplicates":                          # some entries twice, in one part of the rows
        at = np.sort(rng.choice(np.flatnonzero(rows < n // 2), 300, replace=False))
        rows, col = np.insert(rows, at, rows[at]), np.insert(col, at, col[at])
    if kind != "sorted":
        order = np.lexsort((rng.random(len(rows)), rows))
        rows, col = rows[order], col[order]
    rp, col = rebuild(M, rows, col)
    want, _ = oracle.partition(M, N, rp, col)
    assert want["dense_nnz"] > 0 and (not many or max(np.diff(want["nDiasPtr"])) > 32)
    got = tc.Plan.from_csr(M, N, rp, col).export()
    for k in oracle.FORMAT_KEYS:
        assert got[k] == want[k], k
    for k in ("xStart", "yStart", "xStop", "nDiasPtr", "neg_offsets", "csrRow", "csrCol"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


def blocks(nb, side, gap, dup, seed):
    """nb diagonal blocks of seven diagonals with holes, some with entries twice."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for b in range(nb):
        o = b * (side + gap)
        i = np.arange(o, o + side)
        for d in range(-3, 4):
            ok = (i + d >= o) & (i + d < o + side) & (rng.random(side) >= 0.05)
            rows.append(i[ok])
            cols.append(i[ok] + d)
        if b in dup:
            k = o + rng.integers(0, side, 6)
            rows.append(k)
            cols.append(k)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((cols, rows))
    M = nb * (side + gap)
    return (M,) + rebuild(M, rows[order], cols[order])


@pytest.mark.parametrize("nb,height,more_than", [(40, 1024, 32), (270, 4096, 250)])
def test_many_shapes(tc, dev, nb, height, more_than):
    """More shapes than one histogram launch counts, and more claiming shapes
    than there are marks, with duplicate entries in shapes before and after."""
    M, rp, col = blocks(nb, 100, 12, {2, nb // 3, nb - 3}, 1)
    over = dict(thumb_height=height, min_contour=10, min_shape_side=20)
    want, _ = oracle.partition(M, M, rp, col, params=oracle.default_params(**over))
    assert want["dia_shapes"] > more_than and want["zero_elements"] > 0
    got = tc.Plan.from_csr(M, M, rp, col, prm=tc.params(**over)).export()
    for k in oracle.FORMAT_KEYS:
        assert got[k] == want[k], k
    for k in ("xStart", "yStart", "xStop", "nDiasPtr", "neg_offsets", "csrRow", "csrCol"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


def test_more_holes_than_words(tc, dev):
    """Two wide bands of few entries under a density threshold near zero: their
    holes are more than 2^31, which no row pointer holds; refused, and the same
    matrix is partitioned under the usual threshold."""
    import torch
    side, gap, half = 990_000, 60_000, 980
    M = 2 * (side + gap)
    g = torch.Generator(dev).manual_seed(3)
    rows = torch.arange(M, device=dev)
    rows = rows[(rows % (side + gap)) < side].repeat_interleave(4)
    block = torch.div(rows, side + gap, rounding_mode="floor") * (side + gap)
    cols = rows + torch.randint(-half, half + 1, rows.shape, device=dev, generator=g)
    ok = (cols >= block) & (cols < block + side)
    keys = torch.unique(rows[ok] * M + cols[ok])
    rows = torch.div(keys, M, rounding_mode="floor")
    rp = torch.zeros(M + 1, dtype=torch.int64, device=dev)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=M), 0)
    rp, col = rp.int(), (keys - rows * M).int()
    with pytest.raises(tc.TcError) as e:
        tc.Plan.from_csr(M, M, rp, col, prm=tc.params(density=1e-6), on_device=True)
    assert e.value.status == 8 and "2^31" in str(e.value)          # TC_ERR_UNSUPPORTED
    plan = tc.Plan.from_csr(M, M, rp, col, on_device=True)
    assert plan.info()["dia_shapes"] == 0 and plan.info()["nnz_csr"] == col.numel()
