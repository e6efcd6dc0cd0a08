"""The training recurrences at the edges of their blocks of 16 trajectories and
of their paired time steps, against FP64 autograd (oracle/encoder_ref.py).

Tolerances: an operand's three BF16 parts hold all 24 bits and sums of up to
128 products accumulate in FP32 (128 * 2^-24 = 8e-6 of their largest term a
step); the weight gradients' operands have two parts (2^-16 = 1.5e-5 a
product).  Allowed: 1e-4 of the largest gradient, 2e-5 of a prediction."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [
    [1, 1],                      # one point: no recurrent product
    [2, 1, 3],                   # even, odd, a block that is nearly empty
    [7] * 15, [8] * 16, [9] * 17,  # one under, exactly, one over a block; odd and even steps
    list(range(1, 34)),          # every length 1..33: rows of a block that end at each step
    [40] + [1] * 32,             # one long row among short ones, three blocks
], ids=lambda v: f"{len(v)}x{max(v)}")
def test_training_gradients_at_block_edges(lens):
    from oracle import encoder_ref as R
    from trajsimimeasures_b200 import datagen as D
    from trajsimimeasures_b200.engine import TrajSet
    from trajsimimeasures_b200.surrogate import Encoder
    rng = np.random.default_rng(len(lens))
    pts, off, ln = D._walks(rng, np.array(lens), D.STEP_SIGMA)
    trajs = D.unpack(pts, off, ln)
    s = TrajSet.from_lists(trajs)
    enc = Encoder.init(s, seed=21)
    enc.params.mul_(2.0)
    n = len(lens)
    ia, ib = np.arange(n), (np.arange(n) + 1) % n
    y = rng.uniform(0.05, 0.5, n)
    loss, grad, pred = enc.loss_grad(s, np.arange(n), ia, ib, y)
    enc.check_training()
    l_ref, g_ref, p_ref = R.loss_grad(enc.params.cpu().numpy(), trajs, enc.nrm, ia, ib, y)
    np.testing.assert_allclose(pred.cpu().numpy(), p_ref, rtol=2e-5, atol=1e-6)
    assert abs(loss.item() - l_ref) <= 1e-4 * abs(l_ref) + 1e-7
    g = grad.cpu().numpy().astype(np.float64)
    assert np.abs(g - g_ref).max() <= 1e-4 * np.abs(g_ref).max()
    # the same workspace again: nothing of a batch is left over in the next
    assert np.array_equal(enc.loss_grad(s, np.arange(n), ia, ib, y)[2].cpu().numpy(), pred.cpu().numpy())


@pytest.mark.parametrize("n,longest", [(1, 1), (5, 3), (127, 20), (128, 21), (129, 31)])
def test_embedding_in_batches_is_one_by_one(n, longest):
    """Blocks of 128 trajectories, partly filled; odd and even numbers of
    steps: a trajectory's embedding doesn't depend on the batch around it."""
    from trajsimimeasures_b200 import datagen as D
    from trajsimimeasures_b200.engine import TrajSet
    from trajsimimeasures_b200.surrogate import Encoder
    rng = np.random.default_rng(n)
    L = rng.integers(1, longest + 1, n)
    L[-1] = longest
    s = TrajSet.from_lists(D.unpack(*D._walks(rng, L, D.STEP_SIGMA)))
    enc = Encoder.init(s, seed=22)
    e = enc.embed(s, batch=n)
    # (a set of one point has no spread to normalise by: NaN throughout)
    assert bool(torch.isfinite(e).all()) == bool(np.isfinite(enc.nrm).all())
    again = enc.embed(s, batch=max(1, n // 3))
    np.testing.assert_array_equal(again.cpu().numpy(), e.cpu().numpy())
