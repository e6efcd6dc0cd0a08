"""The DTW, ERP and discrete Frechet matrix kernels on both sides of their
dispatch line (query length 96) and at the edges of their strips of 16 and 8
rows: plain, symmetric and gather forms bit-identical to the FP32 twin in exact
mode, a bad length included."""
import numpy as np
import pytest

from trajsimimeasures_b200 import datagen as D

pytestmark = pytest.mark.gpu
G = (-8.625, 41.15)
MID = {"dtw": 0, "erp": 3, "dfrechet": 4}


@pytest.mark.parametrize("measure", ["dtw", "erp", "dfrechet"])
@pytest.mark.parametrize("longest", [3, 96, 97, 200])
@pytest.mark.parametrize("rows", [0, 4, 16])
def test_matrix_forms_equal_the_twin(measure, longest, rows, oracle_mod):
    import torch
    from trajsimimeasures_b200 import engine
    lens = np.array([n for n in (1, 2, 3, 0, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 64, 96, 97, 113, 200)
                     if n <= longest])
    rng = np.random.Generator(np.random.PCG64(31))
    pts, off, lens = D._walks(rng, lens, 2e-4)
    n = len(lens)
    ia, ib = np.repeat(np.arange(n), n), np.tile(np.arange(n), n)
    want = oracle_mod.pairs_idx(oracle_mod.pairs_f32, MID[measure], pts, off, lens, ia, ib, gpoint=G)[0].reshape(n, n)
    s = engine.TrajSet.from_packed(pts, off, lens)
    kw = dict(gpoint=G, exact=True, rows=rows)
    out = torch.full((n, n), 7.0, device="cuda")
    engine.matrix_raw(measure, s, s, out=out, **kw)
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    engine.allpairs_sym_raw(measure, s, out=out, **kw)
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    cand = torch.as_tensor(np.tile(np.arange(n)[::-1].copy(), (n, 1)).astype(np.int32), device="cuda")
    cand[:, 0] = n  # outside the database
    engine.matrix_gather_raw(measure, s, s, cand, out=out, **kw)
    got = out.cpu().numpy()
    assert np.isnan(got[:, 0]).all() and np.array_equal(got[:, 1:], want[:, ::-1][:, 1:], equal_nan=True)
    s.lens[0] = -1  # a bad length: NaN in its row and column, the others untouched
    engine.matrix_raw(measure, s, s, out=out, **kw)
    got = out.cpu().numpy()
    assert np.isnan(got[0]).all() and np.isnan(got[:, 0]).all()
    assert np.array_equal(got[1:, 1:], want[1:, 1:], equal_nan=True)
