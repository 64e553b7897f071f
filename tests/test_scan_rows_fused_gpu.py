"""Row scans over fused producers at the edges of a chunk: rows shorter than, as long as and longer than a
warp's part and a block's chunk, with several rows per block and one."""
import pytest

from helpers import TYPES  # noqa: F401  (the helpers' types name the cases)
from test_map_gpu import run_scan_map
from test_scan_gpu import FLAVOURS
from test_scan_zip_gpu import run_scan_zip

pytestmark = pytest.mark.gpu

SHAPES = [(3, 1), (2, 255), (3000, 513), (2600, 512), (700, 1025), (3, 16_384), (2, 16_385), (500, 4097)]


@pytest.mark.parametrize("t", ["i32", "i64", "f32", "f64"])
@pytest.mark.parametrize("shape", SHAPES)
def test_scan_rows_fused_chunks(acc, orc, dev, t, shape):
    zops = ["+", "*", "min", "max"]
    for i, (d, k) in enumerate(FLAVOURS):
        g = zops[(i + shape[1]) % 4]
        run_scan_zip(acc, orc, dev, t, "max" if i % 2 else "min", g, shape, d, k, offset=i % 2)
        run_scan_map(acc, orc, dev, t, "min" if i % 2 else "max", g, shape, d, k)
    run_scan_zip(acc, orc, dev, t, "+", "+", shape, 0, 0)
    run_scan_zip(acc, orc, dev, t, "+", "*", shape, 1, 1)
