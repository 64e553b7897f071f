"""foldSeg of short segments on either side of the average lengths at which its form changes: compensated sums of
fewer than 11 values a segment, zipped ones of fewer than 16, in one launch and in three, with empty segments."""
import numpy as np
import pytest
import torch

from helpers import TYPES, assert_fold_close, case_rng, gen
from test_fold_zip_gpu import zipped

pytestmark = pytest.mark.gpu


def offsets(n, nseg, rng, kind):
    if kind == "equal":
        return np.round(np.linspace(0, n, nseg + 1)).astype(np.int32)
    cuts = np.sort(rng.integers(0, n + 1, size=nseg - 1))  # many of them empty or of one value
    return np.concatenate([[0], cuts, [n]]).astype(np.int32)


def check(orc, got, z, x, off, dt, op):
    ref, ref64, absum = orc.fold_seg(op, z, x, off), None, None
    if np.dtype(dt).kind == "f":
        c = np.concatenate([[0.0], np.cumsum(x.astype(np.longdouble))])
        a = np.concatenate([[0.0], np.cumsum(np.abs(x.astype(np.longdouble)))])
        ref64 = (z + np.diff(c[off])).astype(np.float64)
        absum = (abs(z) + np.diff(a[off])).astype(np.float64)
    assert_fold_close(got, ref, ref64, absum, dt, op)


@pytest.mark.parametrize("kind", ["equal", "random"])
@pytest.mark.parametrize("nseg,per", [(1, 10), (300, 1), (4000, 3), (4096, 11), (4097, 11), (50_000, 7), (50_000, 11), (20_000, 12)])
@pytest.mark.parametrize("t,lengths", [("f32", False), ("f32", True), ("i32", False)])
def test_foldseg_short(acc, orc, dev, t, lengths, nseg, per, kind):
    dt, n = TYPES[t], nseg * per - (per == 11 and nseg % 2)
    rng = case_rng("short", t, lengths, nseg, per, kind)
    x, off = gen(dt, "+", n, rng), offsets(n, nseg, rng, kind)
    seg = torch.from_numpy(np.diff(off) if lengths else off).to(dev)
    got = acc.fold_seg("+", 5, torch.from_numpy(x).to(dev), seg, offsets=not lengths)
    acc.sync()
    check(orc, got.cpu().numpy(), 5, x, off, dt, "+")


@pytest.mark.parametrize("kind", ["equal", "random"])
@pytest.mark.parametrize("nseg,n", [(1, 15), (1, 40), (500, 7999), (500, 8000), (30_000, 479_999), (30_000, 480_000)])
@pytest.mark.parametrize("t", ["i32", "f32", "f64"])
def test_foldseg_zip_short(acc, orc, dev, t, nseg, n, kind):
    dt = TYPES[t]
    rng = case_rng("short zip", t, nseg, n, kind)
    x, y, off = gen(dt, "+", n, rng), gen(dt, "+", n, rng), offsets(n, nseg, rng, kind)
    with np.errstate(over="ignore"):
        zs = zipped("*", x, y)
    got = acc.fold_seg_zipwith("+", "*", 5, torch.from_numpy(x).to(dev), torch.from_numpy(y).to(dev),
                               torch.from_numpy(off).to(dev))
    acc.sync()
    check(orc, got.cpu().numpy(), 5, zs, off, dt, "+")
