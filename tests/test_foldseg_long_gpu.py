"""foldSeg over segments that span many tiles: alone, beside short ones, one after another, in the first and last
tiles, and of lengths around whole numbers of tiles and of blocks of tiles."""
import numpy as np
import pytest
import torch

from helpers import TYPES, assert_fold_close, case_rng, gen

pytestmark = pytest.mark.gpu

TILE = 8192  # 4-byte values per tile (8-byte types: half)
CASES = {
    "one": [600 * TILE + 5], "whole tiles": [300 * TILE], "short": [3 * TILE + 1, 7, 2 * TILE],
    "around a block of tiles": [256 * TILE - 1, 2, 255 * TILE, TILE, 257 * TILE + 3, 0, 0, 5],
    "past a walk's step": [2304 * TILE + 9, 1], "last tile": [1, 0, 700 * TILE, 3],
    "many": [40 * TILE + 1] * 23 + [3] * 700 + [90 * TILE],
}


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("t,op,prec", [("f32", "+", "default"), ("f32", "+", "plain"), ("i32", "+", "default"),
                                       ("i64", "max", "default"), ("f64", "+", "default"), ("f32", "+", "fp64")])
def test_foldseg_long_segments(acc, orc, dev, t, op, prec, case):
    dt = TYPES[t]
    off = np.concatenate([[0], np.cumsum(CASES[case])]).astype(np.int64)
    x = gen(dt, op, int(off[-1]), case_rng("long", t, op, prec, case))
    z = {"+": 5, "max": -7}[op]
    got = acc.fold_seg(op, z, torch.from_numpy(x).to(dev), torch.from_numpy(off).to(dev), prec=prec)
    acc.sync()
    ref = orc.fold_seg(op, z, x, off)
    ref64 = absum = None
    if np.dtype(dt).kind == "f":
        spans = [(int(u), int(v)) for u, v in zip(off[:-1], off[1:])]
        ref64 = np.array([z + x[u:v].astype(np.float64).sum() for u, v in spans])
        absum = np.array([abs(z) + np.abs(x[u:v].astype(np.float64)).sum() for u, v in spans])
    assert_fold_close(got.cpu().numpy(), ref, ref64, absum, dt, op, prec if prec == "plain" else None)
