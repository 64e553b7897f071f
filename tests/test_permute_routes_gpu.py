"""permute on either side of the numbers of updates from which private bins, and wider loads, are taken."""
import numpy as np
import pytest
import torch

from helpers import TYPES, _diff, case_rng, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,op,const,m,n", [
    ("i64", "+", None, 1000, (1 << 15) - 1), ("i64", "+", None, 1000, 1 << 15), ("i64", "+", 3, 1000, (1 << 15) - 1),
    ("i64", "max", None, 129, 1 << 15), ("i32", "*", None, 4000, (1 << 15) - 3), ("u32", "*", None, 4000, 1 << 15),
    ("f32", "+", None, 5000, (1 << 18) - 1), ("f32", "+", None, 5000, 1 << 18), ("f32", "+", None, 512, 1 << 16),
    ("f32", "+", None, 513, 1 << 16), ("f32", "+", 0.5, 64, (1 << 16) - 1), ("f64", "+", None, 3000, (1 << 20) - 1),
    ("f64", "+", None, 3000, 1 << 20), ("f32", "min", None, 1000, 64_000), ("f32", "max", None, 1000, 63_999),
    ("f64", "max", None, 1000, 128_000), ("f64", "min", None, 1000, 127_999), ("f32", "max", None, 30_000, (1 << 19) - 1),
    ("f32", "max", None, 30_000, (1 << 19) + 3), ("f32", "*", None, 77, 1 << 15), ("f64", "*", None, 77, (1 << 15) - 1),
])
@pytest.mark.parametrize("keys", ["uniform", "hot", "sorted"])
def test_permute_routes(acc, orc, dev, t, op, const, m, n, keys):
    dt = TYPES[t]
    rng = case_rng("routes", t, op, const, m, n, keys)
    idx = rng.integers(-1, m, size=n).astype(np.int32)
    if keys == "hot":
        idx[rng.random(n) < 0.7] = m // 3
    elif keys == "sorted":
        idx = np.sort(idx)
    xs = None if const is not None else gen(dt, op, n, rng)
    defaults = gen(dt, op, m, rng)
    got = acc.permute(op, torch.from_numpy(defaults).to(dev), torch.from_numpy(idx).to(dev),
                      const if xs is None else torch.from_numpy(xs).to(dev))
    acc.sync()
    got = got.cpu().numpy()
    if dt in (np.float32, np.float64) and op == "+":
        # one rounding per addition in any order: per bin, additions * eps * sum |x|
        keep = idx >= 0
        src = np.full(n, float(const)) if xs is None else xs.astype(np.float64)
        ref, ab, cnt = defaults.astype(np.float64), np.abs(defaults.astype(np.float64)), np.ones(m)
        np.add.at(ref, idx[keep], src[keep])
        np.add.at(ab, idx[keep], np.abs(src[keep]))
        np.add.at(cnt, idx[keep], 1.0)
        assert np.all(np.abs(got - ref) <= cnt * np.finfo(dt).eps * ab + 1e-30)
    else:
        ref = orc.permute(op, defaults, idx, xs, cval=const)
        same = (got == ref) | ((got != got) & (ref != ref))
        assert same.all(), _diff(got, ref)
