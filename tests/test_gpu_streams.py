"""Calls with stream=: what they gather and launch follows the current stream's
work so far, all of it on the given stream (here the indices are written late,
behind a long-running kernel), and results equal those of the default stream."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu


def _late(values, first):
    """A device tensor that holds `first` until a kernel of about 0.1 s is through."""
    import torch
    buf = torch.full_like(values, first)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)
    buf.copy_(values)
    return buf


def _set(n, hi, seed):
    from trajsimimeasures_b200 import engine
    rng = np.random.Generator(np.random.PCG64(seed))
    return engine.TrajSet.from_packed(*D._walks(rng, rng.integers(2, hi + 1, n), 2e-4))


@pytest.mark.parametrize("measure", ["dtw", "hausdorff", "edr"])
def test_index_pairs(measure):
    import torch
    from trajsimimeasures_b200 import engine
    s = _set(500, 60, 1)
    rng = np.random.default_rng(2)
    ia, ib = (torch.as_tensor(rng.integers(0, s.n, 40000), device="cuda") for _ in range(2))
    want = engine.pairs_in_set(measure, s, ia, ib, eps=3e-4, order=torch.arange(40000, dtype=torch.int32, device="cuda"))[0]
    side = torch.cuda.Stream()
    la, lb = _late(ia, 0), _late(ib, 0)
    got, _ = engine.pairs_in_set(measure, s, la, lb, eps=3e-4, stream=side)
    del la, lb
    junk = [torch.full((40000,), -1, dtype=torch.int64, device="cuda") for _ in range(4)]
    side.synchronize()
    assert torch.equal(got, want) and len(junk) == 4


@pytest.mark.parametrize("longest", [60, 1500])  # the gather form, and queries too long for it
def test_knn_rerank_and_exhaustive(longest):
    import torch
    from trajsimimeasures_b200 import engine, knn
    d = _set(300, 60, 3)
    rng = np.random.Generator(np.random.PCG64(4))
    q = engine.TrajSet.from_packed(*D._walks(rng, np.r_[5, 9, longest], 2e-4))
    cand = torch.as_tensor(np.stack([rng.permutation(300)[:200] for _ in range(3)]), device="cuda")
    want = knn.knn_rerank(q, d, cand, 7)
    side = torch.cuda.Stream()
    got = knn.knn_rerank(q, d, _late(cand, 0), 7, stream=side)
    side.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    if longest <= 1400:
        want = knn.knn_exhaustive(q, d, 7, chunk=100)
        pts = d.pts.clone()
        d.pts = _late(pts, 0.0)
        got = knn.knn_exhaustive(q, d, 7, chunk=100, stream=side)
        side.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_matrix_many():
    import torch
    from trajsimimeasures_b200 import core, engine
    rng = np.random.Generator(np.random.PCG64(5))
    s = engine.TrajSet.from_packed(*D._walks(rng, np.r_[rng.integers(2, 60, 50), 1500], 2e-4))
    ms = ["dtw", "edr", "lcss", "hausdorff"]
    want = core.matrix_many(ms, s, None, s, None, eps=3e-4)
    side = torch.cuda.Stream()
    s.pts = _late(s.pts.clone(), 0.0)
    got = core.matrix_many(ms, s, None, s, None, eps=3e-4, stream=side)
    assert all(np.array_equal(got[m], want[m], equal_nan=True) for m in ms)
