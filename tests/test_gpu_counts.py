"""EDR and LCSS counts of the bit-vector kernels against the FP32 twin, equal
on every pair: at the edges of their 32-row words, with matches nowhere, in
places and nearly everywhere, with non-finite coordinates, and at the ends of
the threshold's range."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu
EDGES = [0, 1, 2, 5, 31, 32, 33, 40, 63, 64, 65, 95, 96, 97, 128, 200, 255, 256, 257]
MID = {"edr": 1, "lcss": 2}


def _set(kind, seed=21):
    rng = np.random.Generator(np.random.PCG64(seed))
    pts, off, lens = D._walks(rng, np.asarray(EDGES), 2e-4)
    if kind != "apart":  # every trajectory starts at the first one's start
        first = pts[off[1]].copy()
        for k in range(len(EDGES)):
            if EDGES[k]:
                pts[off[k]:off[k] + lens[k]] += first - pts[off[k]]
    if kind == "dense":
        pts = (first + rng.normal(0, 1e-4, pts.shape)).astype(np.float32)
    if kind == "special":
        for k in range(3, len(lens), 3):
            pts[off[k] + lens[k] // 2, k % 2] = [np.nan, np.inf, -np.inf][k % 3]
            pts[off[k] + lens[k] // 3] = np.nan
    return pts, off, lens


def _all_pairs(n):
    return np.repeat(np.arange(n), n), np.tile(np.arange(n), n)


def _check(out, cnt, want, want_cnt):
    assert np.array_equal(np.asarray(cnt), want_cnt)
    assert np.array_equal(np.asarray(out, np.float32), want, equal_nan=True)


@pytest.mark.parametrize("measure", ["edr", "lcss"])
@pytest.mark.parametrize("kind,eps", [("apart", 3e-4), ("meeting", 3e-4), ("dense", 1.5e-4), ("special", 3e-4),
                                      ("meeting", 0.0), ("meeting", 1e-22), ("meeting", 1.0), ("dense", 1e30)])
def test_counts_equal_the_twin(measure, kind, eps, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine, sched
    pts, off, lens = _set(kind)
    n = len(lens)
    ia, ib = _all_pairs(n)
    want, want_cnt = oracle_mod.pairs_idx(oracle_mod.pairs_f32, MID[measure], pts, off, lens, ia, ib, eps=eps)
    s = engine.TrajSet.from_packed(pts, off, lens)
    out, cnt = engine.matrix(measure, s, s, eps=eps)
    _check(out.cpu(), cnt.cpu(), want.reshape(n, n), want_cnt.reshape(n, n))
    engine.allpairs_sym_raw(measure, s, out=out, counts=cnt, eps=eps)
    _check(out.cpu(), cnt.cpu(), want.reshape(n, n), want_cnt.reshape(n, n))
    cand = torch.as_tensor(np.tile(np.arange(n)[::-1].copy(), (n, 1)).astype(np.int32), device="cuda")
    engine.matrix_gather_raw(measure, s, s, cand, out=out, counts=cnt, eps=eps)
    _check(out.cpu(), cnt.cpu(), want.reshape(n, n)[:, ::-1], want_cnt.reshape(n, n)[:, ::-1])
    out, cnt = engine.pairs_in_set(measure, s, np.tile(ia, 30), np.tile(ib, 30), eps=eps)  # not a small batch
    _check(out.cpu(), cnt.cpu(), np.tile(want, 30), np.tile(want_cnt, 30))
    ta, tb = torch.as_tensor(ia, device="cuda"), torch.as_tensor(ib, device="cuda")
    p = sched.PairsScheduler(s.pts, s.off[ta], s.lens[ta], s.off[tb], s.lens[tb], [measure], eps=eps)
    p.run()
    _check(p.out[MID[measure]].cpu(), p.counts[MID[measure]].cpu(), want, want_cnt)


def test_scheduled_counts_with_the_least_shared_memory(oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine, sched
    pts, off, lens = _set("meeting")
    one = np.flatnonzero(np.asarray(EDGES) == 1)[0]
    ia, ib = np.full(len(lens), one), np.arange(len(lens))
    want, want_cnt = oracle_mod.pairs_idx(oracle_mod.pairs_f32, MID["edr"], pts, off, lens, ia, ib, eps=3e-4)
    s = engine.TrajSet.from_packed(pts, off, lens)
    ta, tb = torch.as_tensor(ia, device="cuda"), torch.as_tensor(ib, device="cuda")
    p = sched.PairsScheduler(s.pts, s.off[ta], s.lens[ta], s.off[tb], s.lens[tb], ["edr"], eps=3e-4, warp_floats=32)
    p.run()
    _check(p.out[1].cpu(), p.counts[1].cpu(), want, want_cnt)
