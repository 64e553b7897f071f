"""foldSeg of many segments on either side of the number of tiles up to which the last tile completes the segments
that cross tiles, with crossing segments at every tile's edge and segments of many tiles."""
import numpy as np
import pytest
import torch

from helpers import TYPES, assert_fold_close, case_rng, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,op,prec", [("i32", "+", "default"), ("i64", "max", "default"), ("f32", "+", "default"),
                                       ("f32", "+", "fp64"), ("f64", "+", "default")])
@pytest.mark.parametrize("tiles", [1, 33, 127, 128, 129, 255, 256, 257])
@pytest.mark.parametrize("mean", [3, 40])
def test_foldseg_finish(acc, orc, dev, t, op, prec, tiles, mean):
    dt = TYPES[t]
    rng = case_rng("finish", t, op, prec, tiles, mean)
    tile = 32768 // np.dtype(dt).itemsize
    n = (tiles - 1) * tile + int(rng.integers(1, tile))
    off = np.sort(rng.integers(0, n + 1, size=max(n // mean, 4200)))
    if tiles > 40:  # one segment of some 30 tiles
        off = off[(off < 5 * tile + 3) | (off > 35 * tile + 1)]
    off = np.concatenate([[0], off, [n]]).astype(np.int32)
    x = gen(dt, op, n, rng)
    z = {"+": 5, "max": -7}[op]
    ref = orc.fold_seg(op, z, x, off)
    ref64 = absum = None
    if np.dtype(dt).kind == "f":
        c = np.concatenate([[0.0], np.cumsum(np.abs(x).astype(np.longdouble))])
        s = np.concatenate([[0.0], np.cumsum(x.astype(np.longdouble))])
        ref64 = (z + (s[off[1:]] - s[off[:-1]])).astype(np.float64)
        absum = (abs(z) + (c[off[1:]] - c[off[:-1]])).astype(np.float64)
    xs, os_ = torch.from_numpy(x).to(dev), torch.from_numpy(off).to(dev)
    for _ in range(3):  # the count of finished tiles is zero again after each call
        got = acc.fold_seg(op, z, xs, os_, prec=prec)
        acc.sync()
        assert_fold_close(got.cpu().numpy(), ref, ref64, absum, dt, op, None)
