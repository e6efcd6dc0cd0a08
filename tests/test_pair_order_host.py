"""pair_order_dev and knn.shape_order on lengths in host memory: the order of
pair_order (no kernel is given a host pointer)."""
import numpy as np
import pytest
import torch

from trajsimimeasures_b200 import engine, knn


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("rows", [4, 8, 16])
def test_order_of_host_lengths(dtype, rows):
    rng = np.random.default_rng(rows)
    la, lb = rng.integers(0, 90, 500), rng.integers(0, 90, 500)
    a, b = torch.as_tensor(la).to(dtype), torch.as_tensor(lb).to(dtype)
    want = engine.pair_order(la, lb, rows)
    for order in (engine.pair_order_dev(a, b, rows), knn.shape_order(a, b, rows)):
        assert order.dtype == torch.int32 and not order.is_cuda
        assert np.array_equal(order.numpy(), want)
