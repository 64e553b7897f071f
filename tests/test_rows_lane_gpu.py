"""Many rows of at most 512 bytes: folds and scans with one lane per row, around the row length and the row
count where they begin, with a last warp that is partly empty."""
import pytest

from test_fold_gpu import run_fold
from test_fold_zip_gpu import run_zip
from test_map_gpu import run_fold_map, run_scan_map
from test_scan_gpu import FLAVOURS, run_scan
from test_scan_zip_gpu import run_scan_zip

pytestmark = pytest.mark.gpu

SHAPES = [(4863, 31), (4864, 2), (4864, 128), (4865, 33), (9731, 15), (4870, 6), (9745, 5), (24_576, 48), (25_089, 49),
          (37_000, 72), (37_376, 73), (400_001, 24), (32_777, 64), (33_281, 65)]


@pytest.mark.parametrize("t,op", [("i32", "+"), ("f32", "+"), ("f32", "min"), ("i64", "xor"), ("f64", "max"), ("f64", "+"), ("u32", "*")])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("offset", [0, 1])
def test_rows_lane(acc, orc, dev, t, op, shape, offset):
    run_fold(acc, orc, dev, t, op, shape, seeded=True, offset=offset)
    run_fold(acc, orc, dev, t, op, shape, seeded=False, offset=offset)
    for d, k in FLAVOURS:
        run_scan(acc, orc, dev, t, op, shape, d, k, offset=offset)


@pytest.mark.parametrize("t", ["i32", "f32"])
@pytest.mark.parametrize("shape", [(4865, 33), (9745, 64)])
@pytest.mark.parametrize("offset", [0, 1])
def test_rows_lane_fused(acc, orc, dev, t, shape, offset):
    run_zip(acc, orc, dev, t, "+", "*", shape, True, offset=offset)
    run_fold_map(acc, orc, dev, t, "max", "+", shape, True, offset=offset)
    for d, k in FLAVOURS:
        run_scan_zip(acc, orc, dev, t, "+", "*", shape, d, k, offset=offset)
        run_scan_map(acc, orc, dev, t, "+", "+", shape, d, k, offset=offset)


@pytest.mark.parametrize("t,op,shape", [("i32", "+", (65_537, 128)), ("i32", "+", (66_049, 129)), ("f32", "+", (65_537, 128)),
                                        ("i64", "max", (200_001, 31)), ("i64", "max", (200_001, 32)), ("f32", "+", (100_001, 63))])
def test_rows_lane_large(acc, orc, dev, t, op, shape):
    # above the size of the segmented pass, which the short rows of scanl / scanr and of scanl' / scanr' leave
    for d, k in FLAVOURS:
        run_scan(acc, orc, dev, t, op, shape, d, k)


@pytest.mark.parametrize("t,op", [("i32", "+"), ("f32", "*"), ("f32", "+"), ("i64", "min"), ("f64", "+"), ("f64", "max")])
@pytest.mark.parametrize("shape", [(9728, 17), (9735, 31), (9736, 32), (9727, 33), (9729, 64), (9730, 96), (9731, 97), (9732, 112),
                                   (9733, 113), (9734, 200), (9735, 201), (77_827, 80)])
def test_rows_by_eights(acc, orc, dev, t, op, shape):
    # a warp folds eight rows at a time: whole and partial steps of 32 values, one to eight rows in the last warp
    for prec in ("default", "plain") if (t, op) == ("f32", "+") else (None,):
        run_fold(acc, orc, dev, t, op, shape, seeded=True, prec=prec)
    run_fold(acc, orc, dev, t, op, shape, seeded=False, offset=1)
    if op == "+":
        run_zip(acc, orc, dev, t, "+", "*", shape, True, offset=1)
        run_fold_map(acc, orc, dev, t, "+", "*", shape, True)
