"""Folds of short rows start from their seed: sums that leave the type's range without it stay in range."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner", [5, 6, 9, 16])
@pytest.mark.parametrize("outer", [300, 9000])
@pytest.mark.parametrize("prec", ["compensated", "plain", "fp64"])
def test_fold_short_rows_from_the_seed(acc, dev, inner, outer, prec):
    e = 2.0 ** 125  # eight of it are out of range; sums of its small multiples are exact
    x = np.zeros((outer, inner), np.float32)
    x[:, 1] = 5 * e
    x[:, inner - 1] = 6 * e
    got = acc.fold("+", float(np.float32(-7 * e)), torch.from_numpy(x).to(dev), prec=prec)
    acc.sync()
    assert np.array_equal(got.cpu().numpy(), np.full(outer, np.float32(4 * e)))
