"""tsm_pair_order: a permutation in non-increasing order of the pairs' classes,
over one CTA and many, with lengths at the edges of the classes and bad ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _side(n):
    n = np.maximum(n, 0)
    e = np.floor(np.log2(np.maximum(n, 1))).astype(int)
    return np.where(n <= 256, (n + 7) // 8, np.minimum(63, 33 + (e - 8) * 8 + ((n >> np.maximum(e - 3, 0)) & 7)))


@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 700_001])
@pytest.mark.parametrize("hi", [3, 300, 40000])
def test_order_is_a_permutation_largest_first(n, hi):
    import torch
    from trajsimimeasures_b200 import engine
    rng = np.random.default_rng(n + hi)
    la, lb = rng.integers(-1, hi + 1, n), rng.integers(0, hi + 1, n)
    la[: min(n, 4)] = [256, 257, 4095, 2**31 - 1][: min(n, 4)]
    o = engine.pair_order_dev(torch.as_tensor(la, dtype=torch.int32, device="cuda"),
                              torch.as_tensor(lb, dtype=torch.int32, device="cuda")).cpu().numpy()
    assert np.array_equal(np.sort(o), np.arange(n))
    key = (_side(np.maximum(la, lb)) * 64 + _side(np.minimum(la, lb)))[o]
    assert (np.diff(key) <= 0).all()
