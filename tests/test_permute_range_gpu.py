"""permute of floats whose updates leave the type's range when they are combined apart from the target's own
value: every order of one-by-one updates of these targets stays in range and gives one result."""
import ctypes

import numpy as np
import pytest
import torch

from helpers import case_rng

pytestmark = pytest.mark.gpu

CODES = {np.float32: 3, np.float64: 4}


def keyed(groups, m, n, rng):
    """Keys, and the places of the listed values of bins 0, 1, ...: side by side, so that one block of threads
    takes them all; the other updates go to the other bins."""
    at = 64 * int(rng.integers(0, n // 64 - 1)) + rng.permutation(64)
    keys, k = rng.integers(len(groups), m, size=n).astype(np.int32), 0
    for b, (_, values) in enumerate(groups):
        for _ in values:
            keys[at[k]] = b
            k += 1
    return keys, at


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("m,n", [(9, 300_000), (3000, 300_003), (3001, 2_000_000)])
@pytest.mark.parametrize("off", [0, 1])
def test_permute_add_keeps_range(acc, dev, dt, m, n, off):
    big = float(np.finfo(dt).max)
    # (target, updates): whole multiples of max / 8, exact in any order from the target on
    e = big / 8
    groups = [(-7 * e, [5 * e, 4 * e, 4 * e]), (7 * e, [-5 * e, -4 * e, -4 * e]), (-np.inf, [6 * e, 6 * e]),
              (3 * e, [np.inf, 6 * e]), (0.0, [np.nan, 1.0]), (0.0, [np.inf, -np.inf]), (-6 * e, [6 * e, 6 * e])]
    rng = case_rng("range+", str(dt), m, n, off)
    keys, at = keyed(groups, m, n, rng)
    vals = np.ones(n, dt)
    target = np.zeros(m, dt)
    k = 0
    for b, (t, values) in enumerate(groups):
        target[b] = t
        for v in values:
            vals[at[k]] = v
            k += 1
    ref = target.astype(np.float64) if dt == np.float32 else target.astype(np.longdouble)
    with np.errstate(invalid="ignore"):
        np.add.at(ref, keys, vals.astype(ref.dtype))
    buf = torch.zeros(m + off, dtype=torch.from_numpy(target).dtype, device=dev)
    buf[off:] = torch.from_numpy(target).to(dev)  # off 1: the target is not on a 16-byte boundary
    src, idx = torch.from_numpy(vals).to(dev), torch.from_numpy(keys).to(dev)
    st = acc.lib().acc_permute(0, CODES[dt], src.data_ptr(), None, idx.data_ptr(), 0, buf[off:].data_ptr(), n, m,
                               torch.cuda.current_stream().cuda_stream)
    assert st == 0
    acc.sync()
    got = buf[off:].cpu().numpy()
    # the other bins count ones: whole numbers below 2^24
    assert np.array_equal(got, ref.astype(dt), equal_nan=True)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("m,n", [(9, 300_000), (3000, 300_003)])
@pytest.mark.parametrize("const", [False, True])
def test_permute_mul_keeps_range(acc, dev, dt, m, n, const):
    p = float(2 ** 60 if dt == np.float32 else 2 ** 500)
    lim = p * p  # 2^120, 2^1000
    fine = float(1 + 2 * np.finfo(dt).eps)
    groups = [(1 / lim, [p, p, p, p]), (lim, [1 / p] * 4), (0.0, [p, p, p]), (lim, [fine / p, 1 / p, 1 / p]),
              (2.0, [0.0, p]), (1.0, [np.inf, 2.0]), (1.0, [np.nan, p]), (-1 / lim, [p, -p, p, p])]
    if const:  # one constant, all bins hit the same number of times or not at all
        groups = [(1 / lim, [p] * 4), (0.0, [p] * 4), (-1 / lim, [p] * 3)]
    rng = case_rng("range*", str(dt), m, n, const)
    keys, at = keyed(groups, m, n, rng)
    vals = np.ones(n, dt)
    target = rng.choice(np.array([0.5, 1.0, -3.0], dt), size=m)
    k = 0
    for b, (t, values) in enumerate(groups):
        target[b] = t
        for v in values:
            vals[at[k]] = v
            k += 1
    if const:
        keys[keys >= len(groups)] = -1  # only the listed bins are updated
    ref = target.astype(np.longdouble)
    with np.errstate(invalid="ignore"):
        for i in np.flatnonzero((keys >= 0) & (keys < len(groups))):
            ref[keys[i]] = ref[keys[i]] * np.longdouble(vals[i])
    c = ctypes.c_float(p) if dt == np.float32 else ctypes.c_double(p)
    out = torch.from_numpy(target).to(dev)
    src, idx = torch.from_numpy(vals).to(dev), torch.from_numpy(keys).to(dev)
    st = acc.lib().acc_permute(1, CODES[dt], None if const else src.data_ptr(), ctypes.byref(c) if const else None,
                               idx.data_ptr(), 0, out.data_ptr(), n, m,
                               torch.cuda.current_stream().cuda_stream)
    assert st == 0
    acc.sync()
    assert np.array_equal(out.cpu().numpy(), ref.astype(dt), equal_nan=True)
