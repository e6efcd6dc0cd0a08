"""The pruned Hausdorff kernels against the FP32 twin (bit for bit in exact
mode), at the edges of their groups, boxes and length classes, and on inputs
that leave them nothing to prune or no finite bound."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu
EDGES = [0, 1, 2, 3, 8, 9, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, 1100]


def _walks(lens, seed, jump=None):
    rng = np.random.Generator(np.random.PCG64(seed))
    pts, off, lens = D._walks(rng, np.asarray(lens), 2e-4)
    if jump:  # no spatial order at all
        pts = rng.uniform(0.0, jump, size=pts.shape).astype(np.float32)
    return pts, off, lens


def _special(pts, off, lens):
    """Non-finite coordinates and coincident points in some trajectories."""
    pts = pts.copy()
    for k in range(3, len(lens), 7):
        if lens[k] > 2:
            pts[off[k] + lens[k] // 2, k % 2] = [np.nan, np.inf, -np.inf][k % 3]
    for k in range(5, len(lens), 7):
        pts[off[k]:off[k] + lens[k]] = pts[off[k]] if lens[k] else 0
    return pts


def _twin(oracle_mod, pts, off, lens, ia, ib):
    return oracle_mod.pairs_f32(5, pts, off[ia], lens[ia], off[ib], lens[ib])[0]


def _same(got, want):
    assert np.array_equal(np.asarray(got, np.float32).view(np.int32), np.asarray(want, np.float32).view(np.int32))


@pytest.mark.parametrize("kind", ["walk", "scattered", "special"])
def test_matrix_and_symmetric_forms_equal_the_twin(kind, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    lens = [n for n in EDGES if n <= 600]
    pts, off, lens = _walks(lens, 11, 0.01 if kind == "scattered" else None)
    if kind == "special":
        pts = _special(pts, off, lens)
    n = len(lens)
    s = engine.TrajSet.from_packed(pts, off, lens)
    ia, ib = np.repeat(np.arange(n), n), np.tile(np.arange(n), n)
    want = _twin(oracle_mod, pts, off, lens, ia, ib).reshape(n, n)
    out = torch.empty((n, n), dtype=torch.float32, device="cuda")
    engine.matrix_raw("hausdorff", s, s, out=out, exact=True)
    _same(out.cpu().numpy(), want)
    engine.allpairs_sym_raw("hausdorff", s, out=out, exact=True)
    _same(out.cpu().numpy(), want)
    cand = torch.as_tensor(np.tile(np.arange(n)[::-1].copy(), (n, 1)).astype(np.int32), device="cuda")
    engine.matrix_gather_raw("hausdorff", s, s, cand, out=out, exact=True)
    _same(out.cpu().numpy(), want[:, ::-1])


@pytest.mark.parametrize("kind", ["walk", "scattered", "special"])
@pytest.mark.parametrize("copies", [1, 30])  # a small batch, and one of more than 64 pairs per SM
def test_pairs_equal_the_twin(kind, copies, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    pts, off, lens = _walks(EDGES, 12, 0.01 if kind == "scattered" else None)
    if kind == "special":
        pts = _special(pts, off, lens)
    n = len(lens)
    s = engine.TrajSet.from_packed(pts, off, lens)
    ia, ib = np.repeat(np.arange(n), n), np.tile(np.arange(n), n)
    want = _twin(oracle_mod, pts, off, lens, ia, ib)
    got, _ = engine.pairs_in_set("hausdorff", s, np.tile(ia, copies), np.tile(ib, copies), exact=True)
    _same(got.cpu().numpy(), np.tile(want, copies))
