"""Row-streaming stencils at the edges of their strips and row ranges, bit-exact against the oracle: widths
around a warp's strip with and without 16-byte rows, arrays thinner than the halo, every boundary."""
import numpy as np
import pytest
import torch

from helpers import _diff, case_rng

pytestmark = pytest.mark.gpu

TYPES = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}
SHAPES = [(1, 128), (2, 127), (3, 64), (25, 132), (41, 129), (23, 260), (64, 513), (61, 1), (40, 2), (700, 388), (1, 20_001)]


@pytest.mark.parametrize("t", list(TYPES))
@pytest.mark.parametrize("pattern", [(3, 3), (1, 3), (3, 1), (5, 5)])
@pytest.mark.parametrize("shape", SHAPES)
def test_stencil_rows(acc, orc, dev, t, pattern, shape):
    rng = case_rng("rows", t, pattern, shape)
    dt = np.dtype(TYPES[t])
    for b in range(4):
        for off in (0, 1):  # off 1: the rows start one element past a 16-byte boundary
            n = shape[0] * shape[1]
            if dt.kind == "f":
                x, w, c = rng.random(n + off).astype(dt), rng.uniform(-1, 1, size=pattern).astype(dt), 0.75
            else:
                x, w, c = (rng.integers(-1000, 1000, size=n + off).astype(dt),
                           rng.integers(1, 4, size=pattern).astype(dt), 7)
            if b == 1:  # a pattern with zero weights; for 3 x 3 the cross
                w[0, 0] = w[-1, -1] = w[0, -1] = w[-1, 0] = 0
            xs = torch.from_numpy(x).to(dev)[off:].view(shape)
            got = acc.stencil(w.tolist(), xs, b, cval=c).cpu().numpy()
            ref = orc.stencil2d(w, x[off:].reshape(shape), b, cval=c)
            assert np.array_equal(got, ref), f"boundary {b} offset {off}: {_diff(got, ref)}"
