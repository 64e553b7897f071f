"""permute through private bins and counters in shared memory, at the edges of their dispatch: the
largest targets of each counter width and the next larger, 64-bit indices, element-wise (unaligned)
reads, remainders, and keys that many lanes of a warp share."""
import numpy as np
import pytest
import torch

from helpers import TYPES, _diff, case_rng, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,op,const,m,n,idx_t,off", [
    ("i32", "+", -7, 57_856, 300_001, np.int32, 0),   # the largest target of 32-bit counters
    ("u32", "+", 5, 57_857, 300_003, np.int32, 0),    # 16-bit counters, an odd bin count
    ("i64", "+", -3, 115_712, 500_000, np.int64, 0),  # the largest target of 16-bit counters
    ("i32", "+", 9, 115_713, 500_001, np.int32, 0),   # the next larger
    ("i32", "+", 3, 65_536, 300_002, np.int32, 1),    # indices not 16-byte aligned
    ("i64", "+", 2, 1, 200_000, np.int64, 0),         # one bin
    ("i64", "+", None, 28_928, 200_003, np.int32, 0), # private 64-bit bins, carries between their halves
    ("i64", "xor", None, 28_929, 200_003, np.int64, 0),
    ("i64", "min", None, 300, 200_001, np.int64, 1),
    ("f32", "+", None, 57_856, 300_002, np.int32, 1),
    ("f32", "+", None, 57_857, 300_002, np.int32, 0),
    ("f32", "+", 0.5, 1000, 9000, np.int64, 0),
    ("f64", "max", None, 28_928, 200_003, np.int32, 0),
    ("u32", "max", None, 57_856, 300_001, np.int32, 3),
])
@pytest.mark.parametrize("hot", [0.0, 0.6])
def test_permute_private(acc, orc, dev, t, op, const, m, n, idx_t, off, hot):
    dt = TYPES[t]
    rng = case_rng("private", t, op, const, m, n, off, hot)
    idx = rng.integers(-2, m, size=n + off).astype(idx_t)
    idx[rng.random(n + off) < hot] = m // 2
    idx[off:][-1] = m - 1
    xs = None if const is not None else gen(dt, op, n + off, rng)
    defaults = gen(dt, op, m, rng)
    src = const if xs is None else torch.from_numpy(xs).to(dev)[off:]
    got = acc.permute(op, torch.from_numpy(defaults).to(dev), torch.from_numpy(idx).to(dev)[off:], src)
    acc.sync()
    got, idx = got.cpu().numpy(), idx[off:]
    xs = None if xs is None else xs[off:]
    if dt in (np.float32, np.float64) and op == "+":
        # one rounding per addition in any order: per bin, additions * eps * sum |x|
        keep = idx >= 0
        src64 = np.full(n, float(const)) if xs is None else xs.astype(np.float64)
        ref, ab, cnt = defaults.astype(np.float64), np.abs(defaults.astype(np.float64)), np.ones(m)
        np.add.at(ref, idx[keep], src64[keep])
        np.add.at(ab, idx[keep], np.abs(src64[keep]))
        np.add.at(cnt, idx[keep], 1.0)
        assert np.all(np.abs(got - ref) <= cnt * np.finfo(dt).eps * ab + 1e-30)
    else:
        ref = orc.permute(op, defaults, idx, xs, cval=const)
        same = (got == ref) | ((got != got) & (ref != ref))
        assert same.all(), _diff(got, ref)


def test_permute_private_out_of_range(acc, dev):
    # a 64-bit index far past the target, and one past it, on the counter and the private kernels
    idx = torch.tensor([0, 3, 4, 1 << 40] + [1] * 60, dtype=torch.int64, device=dev)
    for src in (1, torch.ones(64, dtype=torch.int32, device=dev)):
        out = acc.permute("+", torch.zeros(4, dtype=torch.int32, device=dev), idx, src)
        with pytest.raises(acc.AccError) as e:
            acc.sync()
        assert e.value.status == 7
        assert out.cpu().tolist() == [1, 60, 0, 1]


def test_permute_private_leaves_untouched_bins(acc, dev):
    # bins that no index names keep their bits: subnormals, negative zero, NaN
    tiny = torch.tensor([1e-40, -0.0, float("nan"), 1.0, -3e-42, 2.0, 0.0, 5.0, 1e-45], device=dev)
    idx = torch.tensor([3, 5] * 40, dtype=torch.int32, device=dev)
    out = acc.permute("+", tiny, idx, torch.ones(80, device=dev))
    acc.sync()
    keep = [0, 1, 2, 4, 6, 7, 8]
    assert torch.equal(out[keep].view(torch.int32), tiny[keep].view(torch.int32))
    assert out[[3, 5]].tolist() == [41.0, 42.0]
