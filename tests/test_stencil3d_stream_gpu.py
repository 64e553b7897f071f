"""Plane-streaming 3 x 3 x 3 stencils at the edges of their tiles, bit-exact against the oracle: widths and
heights around a tile's with and without 16-byte rows, one-element extents, every boundary."""
import numpy as np
import pytest
import torch

from helpers import _diff, case_rng

pytestmark = pytest.mark.gpu

TYPES = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}
SHAPES = [(1, 1, 1), (2, 1, 65), (9, 17, 64), (3, 16, 63), (4, 15, 66), (5, 33, 68), (19, 2, 128), (7, 50, 131)]


@pytest.mark.parametrize("t", list(TYPES))
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("pat", ["dense", "star", "mask"])
def test_stencil3d_stream(acc, orc, dev, t, shape, pat):
    rng = case_rng("stream", t, shape, pat)
    dt = np.dtype(TYPES[t])
    n = int(np.prod(shape))
    for b in range(4):
        for off in (0, 1):  # off 1: the rows start one element past a 16-byte boundary
            if dt.kind == "f":
                x, w, c = rng.random(n + off).astype(dt), rng.uniform(-1, 1, size=(3, 3, 3)).astype(dt), 0.75
            else:
                x, w, c = rng.integers(-1000, 1000, size=n + off).astype(dt), rng.integers(1, 4, size=(3, 3, 3)).astype(dt), 7
            if pat == "star":
                keep = np.zeros((3, 3, 3), bool)
                keep[1, 1, :] = keep[1, :, 1] = keep[:, 1, 1] = True
                w[~keep] = 0
            elif pat == "mask":
                w[0, 0, 0] = w[2, 1, 1] = 0
            xs = torch.from_numpy(x).to(dev)[off:].view(shape)
            got = acc.stencil3d(w.tolist(), xs, b, cval=c).cpu().numpy()
            ref = orc.stencil3d(w, x[off:].reshape(shape), b, cval=c)
            assert np.array_equal(got, ref), f"boundary {b} offset {off}: {_diff(got, ref)}"
