"""Batches without a tuning table, one for each launch shape that they choose by themselves: small requests only,
middling ones, large ones, a few folds, and sizes around the widths of the tiles."""
import numpy as np
import pytest
import torch

from helpers import case_rng
from test_batch_gpu import DT, check

pytestmark = pytest.mark.gpu

PLANS = {
    "small": [1, 128, 511, 512, 513, 1024, 1025, 2048, 700, 64] * 4,
    "middling": [2049, 4096, 4097, 16_383, 16_384, 16_385, 70_001, 200_000],
    "large": [262_144, 1_000_003, 5, 2047, 2048, 8192, 32_769, 524_289],
    "many of all": [3, 1000, 5000, 30_000, 65_537, 131_072, 262_143, 300_001] * 6,
}


@pytest.mark.parametrize("plan", list(PLANS))
@pytest.mark.parametrize("kinds", [("fold",), ("scan",), ("fold", "scan")])
def test_batch_default_shapes(acc, orc, dev, plan, kinds):
    rng = case_rng("batch defaults", plan, kinds)
    g = torch.Generator(device=dev)
    g.manual_seed(int(rng.integers(1 << 30)))
    reqs = []
    for i, n in enumerate(PLANS[plan]):
        dt, kind = list(DT.values())[i % 4], kinds[i // 4 % len(kinds)]
        xs = (torch.randn(n, dtype=dt, device=dev, generator=g) if dt.is_floating_point
              else torch.randint(-1000, 1000, (n,), dtype=dt, device=dev, generator=g))
        out = torch.full((1,) if kind == "fold" else (n,), 123, dtype=dt, device=dev)
        reqs.append((kind, xs, out, 7 if i % 3 else None))
    b = acc.Batch("+", reqs)
    for _ in range(2):
        b.launch()
        b.status()
        for kind, xs, out, z in reqs:
            check(orc, out, kind, xs, z, "+")
            out.fill_(9)
    b.close()


@pytest.mark.parametrize("t", list(DT))
@pytest.mark.parametrize("n", [1 << 17, 1 << 20, (1 << 21) + 1])
def test_batch_few_folds(acc, orc, dev, t, n):
    dt = DT[t]
    xs = torch.randint(-100, 100, (n,), device=dev).to(dt)  # whole numbers: exact sums
    out = torch.zeros(1, dtype=dt, device=dev)
    b = acc.Batch("+", [("fold", xs, out, 3)])
    b.launch()
    b.status()
    assert int(out.item()) == int(xs.to(torch.int64).sum().item()) + 3 and np.isfinite(float(out.item()))
    b.close()
