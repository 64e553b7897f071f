"""permute into targets beyond shared memory, on either side of the number of updates from which four are taken per
thread, and with one, two and three updates left over."""
import numpy as np
import pytest
import torch

from helpers import TYPES, _diff, case_rng, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,op", [("i64", "+"), ("i64", "max"), ("i64", "*"), ("i32", "*"), ("f32", "max"), ("f64", "min")])
@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 21) - 1, 1 << 21, (1 << 21) + 3])
@pytest.mark.parametrize("off", [0, 1])
def test_permute_wide(acc, orc, dev, t, op, n, off):
    dt, m = TYPES[t], 500_003
    rng = case_rng("wide", t, op, n, off)
    idx = rng.integers(-1, m, size=n + off).astype(np.int32)
    xs, defaults = gen(dt, op, n + off, rng), gen(dt, op, m, rng)
    got = acc.permute(op, torch.from_numpy(defaults).to(dev), torch.from_numpy(idx).to(dev)[off:],
                      torch.from_numpy(xs).to(dev)[off:])
    acc.sync()
    got, ref = got.cpu().numpy(), orc.permute(op, defaults, idx[off:], xs[off:])
    same = (got == ref) | ((got != got) & (ref != ref))
    assert same.all(), _diff(got, ref)
