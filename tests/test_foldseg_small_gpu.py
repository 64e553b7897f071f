"""Segmented folds around the edges of the one-launch form (all offsets in shared memory: up to 4096 segments,
two tiles per SM) and of the completion across tiles, and short scans around one chunk of the row kernel."""
import numpy as np
import pytest
import torch

from helpers import TYPES, assert_fold_close, case_rng, gen

pytestmark = pytest.mark.gpu


def lengths_of(kind, nseg, n, rng):
    if kind == "one":      # one segment holds everything, over many tiles; the others are empty
        lens = np.zeros(nseg, np.int64)
        lens[nseg // 2] = n
    elif kind == "ends":   # segments end on every tile's last value
        lens = np.full(nseg, 8192, np.int64)
        lens[-1] += n - int(lens.sum())
    else:
        cuts = np.sort(rng.integers(0, n + 1, size=nseg - 1))
        lens = np.diff(np.concatenate([[0], cuts, [n]]))
    return lens


@pytest.mark.parametrize("t,op", [("f32", "+"), ("i32", "max"), ("i64", "+"), ("f64", "+")])
@pytest.mark.parametrize("kind,nseg,n", [("cut", 4096, 300_001), ("cut", 4097, 300_001), ("one", 5, 3_000_003), ("one", 5000, 3_000_003),
                                         ("ends", 40, 40 * 8192), ("ends", 900, 900 * 8192), ("cut", 1, 31), ("cut", 3, 33),
                                         ("cut", 300, 8192 * 304 * 2 + 5)])
@pytest.mark.parametrize("off_t", [np.int32, np.int64])
def test_foldseg_small(acc, orc, dev, t, op, kind, nseg, n, off_t):
    rng = case_rng("small", t, op, kind, nseg, n)
    dt = TYPES[t]
    x = gen(dt, op, n, rng)
    lens = lengths_of(kind, nseg, n, rng)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(off_t)
    z = {"+": 0, "max": np.iinfo(np.int32).min}[op]
    xd = torch.from_numpy(x).to(dev)
    ref = orc.fold_seg(op, z, x, off)
    ref64 = ab = None
    if np.dtype(dt).kind == "f":
        ref64 = orc.fold_seg(op, z, x.astype(np.float64), off)
        ab = orc.fold_seg(op, 0, np.abs(x.astype(np.float64)), off)
    for got in (acc.fold_seg(op, z, xd, torch.from_numpy(off).to(dev)),
                acc.fold_seg(op, z, xd, torch.from_numpy(lens.astype(off_t)).to(dev), offsets=False)):
        acc.sync()
        assert_fold_close(got.cpu().numpy(), ref, ref64, ab, dt, op)


def test_foldseg_small_bad_offsets(acc, dev):
    x = torch.ones(1000, dtype=torch.int32, device=dev)
    for seg, offsets in (([0, 500, 400, 1000], True), ([0, 10, 2000], True), ([-5, 10, 1000], True), ([600, -1, 10], False)):
        acc.fold_seg("+", 0, x, torch.tensor(seg, dtype=torch.int32, device=dev), offsets=offsets)
        with pytest.raises(acc.AccError) as e:
            acc.sync()
        assert e.value.status == 7
    got = acc.fold_seg("+", 0, x, torch.tensor([0, 1, 1000], dtype=torch.int32, device=dev))
    acc.sync()
    assert got.cpu().tolist() == [1, 999]


@pytest.mark.parametrize("t,op", [("i32", "+"), ("f32", "+"), ("f64", "max"), ("u32", "xor"), ("i64", "*")])
@pytest.mark.parametrize("flavour", ["scanl", "scanl1", "scanl_", "scanr", "scanr1", "scanr_"])
def test_scan_rows_chunks(acc, orc, dev, t, op, flavour):
    # one row and a few rows, around a warp's part, a chunk (16,384 or 8192 elements) and several chunks
    from test_scan_gpu import run_scan
    d, k = acc._SCAN_FLAVOURS[flavour]
    per = 16 if np.dtype(TYPES[t]).itemsize == 4 else 8
    for shape in ((1,), (32 * per - 1,), (32 * per + 1,), (1024 * per,), (1024 * per + 1,), (3, 1024 * per + 1), (5, 33 * per),
                  (2, 3 * 1024 * per + 7), (700, 31)):
        run_scan(acc, orc, dev, t, op, shape, d, k)


@pytest.mark.parametrize("t,op", [("f32", "+"), ("i32", "max"), ("i64", "+"), ("f64", "min")])
@pytest.mark.parametrize("zop", ["+", "*", "min", "max"])
@pytest.mark.parametrize("nseg,n,off_a,off_b", [(1, 40, 0, 0), (700, 8192 * 3, 0, 0), (5000, 300_007, 0, 0), (9, 8192 * 700 + 33, 0, 0),
                                                (500, 30_001, 0, 1), (500, 30_001, 1, 1)])
def test_foldseg_zip_tiles(acc, orc, dev, t, op, zop, nseg, n, off_a, off_b):
    # the fused zipWith on the tiled form (both arrays 16-byte aligned) and beside it
    rng = case_rng("ziptiles", t, op, zop, nseg, n, off_a, off_b)
    dt = TYPES[t]
    x, y = gen(dt, "+", n + off_a, rng), gen(dt, "+", n + off_b, rng)
    off = np.concatenate([[0], np.cumsum(lengths_of("cut" if nseg > 1 else "one", nseg, n, rng))]).astype(np.int32)
    z = {"+": 0, "max": np.iinfo(np.int32).min, "min": 7.0}[op]
    got = acc.fold_seg_zipwith(op, zop, z, torch.from_numpy(x).to(dev)[off_a:], torch.from_numpy(y).to(dev)[off_b:],
                               torch.from_numpy(off).to(dev))
    acc.sync()
    with np.errstate(over="ignore"):
        v = {"+": np.add, "*": np.multiply, "min": np.minimum, "max": np.maximum}[zop](x[off_a:], y[off_b:])
    ref = orc.fold_seg(op, z, v, off)
    ref64 = ab = None
    if np.dtype(dt).kind == "f":
        ref64 = orc.fold_seg(op, z, v.astype(np.float64), off)
        ab = orc.fold_seg("+", 0, np.abs(v.astype(np.float64)), off)
    assert_fold_close(got.cpu().numpy(), ref, ref64, ab, dt, op)
