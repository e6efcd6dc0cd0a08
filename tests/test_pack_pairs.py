"""tsm_pack_pairs (host code, no GPU) against NumPy: types, strides, lengths,
origins, and batches large enough for its threads."""
import numpy as np
import pytest

from trajsimimeasures_b200 import _lib, core


def _pack(a1, la, a2, lb, mode, origin=None):
    n, P = len(la), int(la.sum() + lb.sum())
    off = [np.full(n, -1, np.int64) for _ in range(2)]
    ln = [np.full(n, -1, np.int32) for _ in range(2)]
    pts = np.full((P, 2), np.nan, np.float32)
    o = None if origin is None else np.asarray(origin, np.float64)
    rc = _lib.load().tsm_pack_pairs(a1.ctypes.data, a1.strides[0], a1.strides[1], la.ctypes.data, a2.ctypes.data,
                                    a2.strides[0], a2.strides[1], lb.ctypes.data, n, int(a1.dtype == np.float64), mode,
                                    None if o is None else o.ctypes.data, off[0].ctypes.data, off[1].ctypes.data,
                                    ln[0].ctypes.data, ln[1].ctypes.data, pts.ctypes.data, P)
    return rc, off, ln, pts


@pytest.mark.parametrize("n,L", [(1, 1), (7, 13), (5200, 230)])  # the last: about 1.8 million points, several threads
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("layout", ["plain", "wide", "transposed", "reversed"])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_pack_equals_numpy(n, L, dtype, layout, mode):
    rng = np.random.default_rng(n + L)
    def make():
        if layout == "wide":
            return rng.normal(5e6, 1e3, (n, L, 5)).astype(dtype)[:, :, 1:3]
        if layout == "transposed":
            return rng.normal(5e6, 1e3, (L, n, 2)).astype(dtype).transpose(1, 0, 2)
        a = rng.normal(5e6, 1e3, (n, L, 2)).astype(dtype)
        return a[::-1, ::-1] if layout == "reversed" else a
    a1, a2 = make(), make()
    la, lb = (rng.integers(0 if k else max(L - 2, 0), L + 1, n) for k in range(2))
    if n > 5:  # a side and a pair without points, a first point that is not finite
        la[2] = 0
        la[3] = lb[3] = 0
        la[4], a1[4, 0, 0] = 1, np.inf
    o = (5e6, 5e6 + 0.25)
    rc, off, ln, pts = _pack(a1, la, a2, lb, mode, o if mode == 2 else None)
    assert rc == 0
    lens = np.concatenate([la, lb])
    assert np.array_equal(np.concatenate(off), np.cumsum(lens) - lens)
    assert np.array_equal(np.concatenate(ln), lens)
    org = core._pair_origin_of(core._first_points(a1, la), core._first_points(a2, lb), la, lb) if mode == 1 else \
        np.broadcast_to(np.asarray(o) if mode == 2 else np.zeros(2), (n, 2))
    with np.errstate(over="ignore", invalid="ignore"):
        want = [(a[k, :l].astype(np.float64) - org[k]).astype(np.float32) if mode else a[k, :l].astype(np.float32)
                for a, ls in ((a1, la), (a2, lb)) for k, l in enumerate(ls)]
    assert np.array_equal(pts, np.concatenate(want), equal_nan=True)


def test_bad_arguments():
    a, l = np.zeros((2, 3, 2)), np.array([3, 3])
    assert _pack(a, l, a, np.array([3, -1]), 0)[0] == -1
    assert _pack(a, l, a, l, 3)[0] == -1 and _pack(a, l, a, l, 2)[0] == -1
    assert _lib.load().tsm_pack_pairs(None, 0, 0, l.ctypes.data, None, 0, 0, l.ctypes.data, 2, 1, 0, None, None, None, None,
                                      None, None, 0) == -1
    assert b"tsm_pack_pairs" in _lib.load().tsm_last_error()
