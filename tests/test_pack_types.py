"""tsm_pack_pairs on integer arrays and on strided float64 points (host code, no
GPU) against NumPy: converted to float64, translated, rounded once."""
import numpy as np
import pytest

from trajsimimeasures_b200 import _lib, core


@pytest.mark.parametrize("n,L", [(7, 13), (3000, 230)])  # the latter: about 690,000 points, two threads where strided
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float64])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("mode", [1, 2])
def test_pack_equals_numpy(n, L, dtype, strided, mode):
    rng = np.random.default_rng(n + L)
    top = 2 ** 62 if dtype == np.int64 and n < 10 else 10 ** 7  # 64-bit integers that float64 rounds
    def make():
        a = rng.integers(-top, top, (n, L, 5 if strided else 2)).astype(dtype)
        return a[:, :, 1:3] if strided else a
    a1, a2 = make(), make()
    la, lb = (rng.integers(0, L + 1, n) for _ in range(2))
    la[1] = la[2] = lb[2] = 0
    o = np.array([5e6, 5e6 + 0.25])
    P = int(la.sum() + lb.sum())
    off, ln, pts = np.empty(2 * n, np.int64), np.empty(2 * n, np.int32), np.full((P, 2), np.nan, np.float32)
    rc = _lib.load().tsm_pack_pairs(a1.ctypes.data, a1.strides[0], a1.strides[1], la.ctypes.data, a2.ctypes.data,
                                    a2.strides[0], a2.strides[1], lb.ctypes.data, n, core._PACK_TYPES[a1.dtype], mode,
                                    o.ctypes.data if mode == 2 else None, off.ctypes.data, off[n:].ctypes.data,
                                    ln.ctypes.data, ln[n:].ctypes.data, pts.ctypes.data, P)
    assert rc == 0
    f1, f2 = a1.astype(np.float64), a2.astype(np.float64)
    org = core._pair_origin_of(core._first_points(f1, la), core._first_points(f2, lb), la, lb) if mode == 1 else \
        np.broadcast_to(o, (n, 2))
    want = [(a[k, :l] - org[k]).astype(np.float32) for a, ls in ((f1, la), (f2, lb)) for k, l in enumerate(ls)]
    assert np.array_equal(pts, np.concatenate(want))


def test_unknown_type_is_refused():
    a, l = np.zeros((2, 3, 2)), np.array([3, 3])
    off, ln, pts = np.empty(4, np.int64), np.empty(4, np.int32), np.empty((12, 2), np.float32)
    assert _lib.load().tsm_pack_pairs(a.ctypes.data, a.strides[0], a.strides[1], l.ctypes.data, a.ctypes.data, a.strides[0],
                                      a.strides[1], l.ctypes.data, 2, 4, 0, None, off.ctypes.data, off[2:].ctypes.data,
                                      ln.ctypes.data, ln[2:].ctypes.data, pts.ctypes.data, 12) == -1
