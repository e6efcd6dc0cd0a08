"""The rule of engine.pairs_in_set on which batches are worth sorting: long batches
of long trajectories only (no GPU: the SM count is given)."""
import pytest

from trajsimimeasures_b200 import _lib, engine


@pytest.mark.parametrize("m", range(6))
def test_short_batches_and_short_trajectories_keep_their_order(m, monkeypatch):
    monkeypatch.setattr(engine, "_sm_count", lambda device: 148)
    worth = lambda n, longest: engine._worth_sorting(m, n, longest, None)  # noqa: E731
    counts = m in (_lib.EDR, _lib.LCSS)
    assert not worth(0, 200) and not worth(20000, 200)
    assert not worth(200000, 8) and not worth(200000, 20) and not worth(29601, 64)
    assert worth(100000, 200) != counts and worth(60000, 64) != counts
    assert worth(29601, 200) == (m in (_lib.DTW, _lib.ERP, _lib.HAUSDORFF))
