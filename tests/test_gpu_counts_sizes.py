"""EDR and LCSS matrices on both sides of the line between one warp and one lane
per pair (2,960 pairs of at most 64 points, 14,800 of longer ones; half of them in
the symmetric form), and of the boxes' line of 32 points: counts equal to the
FP32 twin's."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("measure", ["edr", "lcss"])
@pytest.mark.parametrize("nq,nd,longest", [(1, 1, 5), (54, 54, 20), (55, 54, 20), (54, 55, 32), (77, 77, 33), (54, 54, 64),
                                           (55, 55, 64), (55, 55, 65), (121, 122, 65), (122, 122, 70), (3, 5000, 40),
                                           (172, 172, 66)])
@pytest.mark.parametrize("eps", [3e-4, 1.0])
def test_matrix_counts_at_the_lines(measure, nq, nd, longest, eps, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    rng = np.random.Generator(np.random.PCG64(nq * 1000 + nd))
    lens = rng.integers(0, longest + 1, max(nq, nd))
    lens[0] = longest
    pts, off, lens = D._walks(rng, lens, 2e-4)
    d = engine.TrajSet.from_packed(pts, off[:nd], lens[:nd])
    q = engine.TrajSet.from_packed(pts, off[:nq], lens[:nq])
    ia, ib = np.repeat(np.arange(nq), nd), np.tile(np.arange(nd), nq)
    want, want_cnt = oracle_mod.pairs_idx(oracle_mod.pairs_f32, {"edr": 1, "lcss": 2}[measure], pts, off, lens, ia, ib,
                                          eps=eps)
    out, cnt = engine.matrix(measure, q, d, eps=eps)
    assert np.array_equal(cnt.cpu().numpy().ravel(), want_cnt)
    assert np.array_equal(out.cpu().numpy().ravel(), want, equal_nan=True)
    if nq == nd:
        out.fill_(7.0)
        cnt.fill_(7)
        engine.allpairs_sym_raw(measure, d, out=out, counts=cnt, eps=eps)
        assert np.array_equal(cnt.cpu().numpy().ravel(), want_cnt)
    cand = torch.as_tensor(np.tile(np.arange(nd)[::-1].copy(), (nq, 1)).astype(np.int32), device="cuda")
    engine.matrix_gather_raw(measure, q, d, cand, out=out, counts=cnt, eps=eps)
    assert np.array_equal(cnt.cpu().numpy()[:, ::-1].ravel(), want_cnt)
