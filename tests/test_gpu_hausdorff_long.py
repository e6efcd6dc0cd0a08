"""The pruned Hausdorff kernels where a trajectory is a CTA's and not one warp's
(above 256 points), alone and among short ones, and where neither fits (the
unpruned kernels): bit-identical to the FP32 twin in exact mode."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu
SHORT = [1, 2, 9, 64, 65, 200]
LONG = [0, 3, 31, 255, 256, 257, 300, 511, 1023, 1025, 2500, 4000]


def _data(lens, kind, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    pts, off, lens = D._walks(rng, np.asarray(lens), 2e-4)
    if kind == "scattered":  # no spatial order: nothing to prune
        pts = rng.uniform(0.0, 0.01, size=pts.shape).astype(np.float32)
    if kind == "special":
        for k in range(1, len(lens), 3):
            if lens[k] > 2:
                pts[off[k] + lens[k] // 2, k % 2] = [np.nan, np.inf, -np.inf][(k // 3) % 3]
    return pts, off, lens


def _same(got, want):
    assert np.array_equal(np.asarray(got, np.float32).view(np.int32), np.asarray(want, np.float32).view(np.int32))


def _twin(O, q, d):
    (qp, qo, ql), (dp, do, dl) = q, d
    pts = np.concatenate([qp, dp])
    ia, ib = np.repeat(np.arange(len(ql)), len(dl)), np.tile(np.arange(len(dl)), len(ql))
    return O.pairs_f32(5, pts, qo[ia], ql[ia], do[ib] + len(qp), dl[ib])[0].reshape(len(ql), len(dl))


@pytest.mark.parametrize("kind", ["walk", "scattered", "special"])
@pytest.mark.parametrize("q_lens,d_lens", [(SHORT, LONG), (LONG, SHORT), (LONG, LONG), ([5, 300, 5000], [7, 400, 6000])],
                         ids=["short-long", "long-short", "long-long", "too-long"])
def test_matrix_and_gather(kind, q_lens, d_lens, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    qd, dd = _data(q_lens, kind, 1), _data(d_lens, kind, 2)
    q, d = engine.TrajSet.from_packed(*qd), engine.TrajSet.from_packed(*dd)
    want = _twin(oracle_mod, qd, dd)
    out = torch.full((q.n, d.n), 7.0, device="cuda")
    engine.matrix_raw("hausdorff", q, d, out=out, exact=True)
    _same(out.cpu().numpy(), want)
    cand = torch.as_tensor(np.tile(np.arange(d.n)[::-1].copy(), (q.n, 1)).astype(np.int32), device="cuda")
    engine.matrix_gather_raw("hausdorff", q, d, cand, out=out, exact=True)
    _same(out.cpu().numpy(), want[:, ::-1])


@pytest.mark.parametrize("kind", ["walk", "scattered", "special"])
def test_symmetric(kind, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    lens = sorted(SHORT + LONG) + [258, 70]
    sd = _data(lens, kind, 3)
    s = engine.TrajSet.from_packed(*sd)
    out = torch.full((s.n, s.n), 7.0, device="cuda")
    engine.allpairs_sym_raw("hausdorff", s, out=out, exact=True)
    _same(out.cpu().numpy(), _twin(oracle_mod, sd, sd))


@pytest.mark.parametrize("kind", ["walk", "scattered", "special"])
@pytest.mark.parametrize("copies", [1, 60])  # a small batch, and one of more than 64 pairs per SM
def test_pairs(kind, copies, oracle_mod):
    from trajsimimeasures_b200 import engine
    sd = _data(LONG + [4096, 4097, 5000], kind, 4)
    s = engine.TrajSet.from_packed(*sd)
    ia, ib = np.repeat(np.arange(s.n), s.n), np.tile(np.arange(s.n), s.n)
    want = _twin(oracle_mod, sd, sd).ravel()
    got, _ = engine.pairs_in_set("hausdorff", s, np.tile(ia, copies), np.tile(ib, copies), exact=True)
    _same(got.cpu().numpy(), np.tile(want, copies))


@pytest.mark.parametrize("n", [9, 60, 150, 300])
@pytest.mark.parametrize("longest", [3, 12, 13, 32, 64])
def test_small_matrices_of_short_trajectories(n, longest, oracle_mod):
    """Both sides of the line between one thread and one warp per pair."""
    import torch
    from trajsimimeasures_b200 import engine
    rng = np.random.default_rng(n)
    sd = _data(np.r_[rng.integers(0, longest + 1, n - 1), longest], "walk", 5)
    s = engine.TrajSet.from_packed(*sd)
    out = torch.full((n, n), 7.0, device="cuda")
    engine.matrix_raw("hausdorff", s, s, out=out, exact=True)
    _same(out.cpu().numpy(), _twin(oracle_mod, sd, sd))
