"""3 x 3 x 3 stencils into an output that starts anywhere an element may: the C entry point takes the caller's
output, which need not lie on the boundary of a wider store (the mirror's own outputs always do)."""
import numpy as np
import pytest
import torch

from helpers import _diff, case_rng

pytestmark = pytest.mark.gpu

TYPES = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}
CODES = {"i32": 0, "i64": 1, "f32": 3, "f64": 4}


@pytest.mark.parametrize("t", list(TYPES))
@pytest.mark.parametrize("shape", [(5, 33, 68), (3, 16, 64), (4, 17, 66), (3, 5, 63), (2, 3, 1)])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_stencil3d_unaligned_output(acc, orc, dev, t, shape, off):
    dt = np.dtype(TYPES[t])
    rng = case_rng("out", t, shape, off)
    n = int(np.prod(shape))
    if dt.kind == "f":
        x, w = rng.random(shape).astype(dt), rng.uniform(-1, 1, size=(3, 3, 3)).astype(dt)
    else:
        x, w = rng.integers(-1000, 1000, size=shape).astype(dt), rng.integers(1, 4, size=(3, 3, 3)).astype(dt)
    xs = torch.from_numpy(x).to(dev)
    buf = torch.full((n + 8,), 77, dtype=xs.dtype, device=dev)
    out = buf[off:off + n]
    assert xs.data_ptr() % 16 == 0 and buf.data_ptr() % 16 == 0
    st = acc.lib().acc_stencil3d(CODES[t], 1, 1, 1, w.ctypes.data, 0, None, xs.data_ptr(), out.data_ptr(), *shape,
                                 torch.cuda.current_stream().cuda_stream)
    assert st == 0
    acc.sync()
    ref = orc.stencil3d(w, x, 0)
    assert np.array_equal(out.cpu().numpy().reshape(shape), ref), _diff(out.cpu().numpy().reshape(shape), ref)
    assert bool((buf[:off] == 77).all()) and bool((buf[off + n:] == 77).all())
