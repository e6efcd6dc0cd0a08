"""The pruned Hausdorff kernels on trajectories of very small extent, where
squared distances are subnormal numbers or underflow: bit-identical to the FP32
twin in exact mode, as everywhere."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu
LENS = [8, 9, 31, 40, 70, 200, 33, 600]


@pytest.mark.parametrize("extent", [1e-22, 1e-20, 1e-19, 1e-17, 1e-15, 1e-13, 1e-9])
def test_tiny_extents_equal_the_twin(extent, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    rng = np.random.Generator(np.random.PCG64(17))
    pts, off, lens = D._walks(rng, np.array(LENS), 2e-4)
    for k in range(len(lens)):  # all from near one place, so that every distance is of the extent's size
        sl = slice(off[k], off[k] + lens[k])
        pts[sl] = (pts[sl] - pts[off[k]]) + rng.uniform(0, 2e-3, 2)
    pts = (pts.astype(np.float64) * (extent / 5e-3)).astype(np.float32)
    n = len(lens)
    ia, ib = np.repeat(np.arange(n), n), np.tile(np.arange(n), n)
    want = oracle_mod.pairs_f32(5, pts, off[ia], lens[ia], off[ib], lens[ib])[0]
    assert (want[ia != ib] > 0).mean() > 0.8
    s = engine.TrajSet.from_packed(pts, off, lens)
    out = torch.empty((n, n), dtype=torch.float32, device="cuda")
    engine.matrix_raw("hausdorff", s, s, out=out, exact=True)
    assert np.array_equal(out.cpu().numpy(), want.reshape(n, n))
    engine.allpairs_sym_raw("hausdorff", s, out=out, exact=True)
    assert np.array_equal(out.cpu().numpy(), want.reshape(n, n))
    for copies in (1, 200):  # a small batch, and one of more than 64 pairs per SM
        got, _ = engine.pairs_in_set("hausdorff", s, np.tile(ia, copies), np.tile(ib, copies), exact=True)
        assert np.array_equal(got.cpu().numpy(), np.tile(want, copies))
