"""Launches whose static and dynamic shared memory exceed the default 48 KB
together but not each alone, each in a process of its own (an earlier launch
with more would leave the kernel's limit raised)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COUNTS = """
import sys
import numpy as np
from oracle import oracle as O
from trajsimimeasures_b200 import datagen as D, engine
m, n, longest = sys.argv[1], int(sys.argv[2]), int(sys.argv[3])
rng = np.random.Generator(np.random.PCG64(9))
pts, off, lens = D._walks(rng, np.r_[rng.integers(1, 7, n - 1), longest], 2e-4)
s = engine.TrajSet.from_packed(pts, off, lens)
_, cnt = engine.matrix(m, s, s, eps=3e-2)
ia = np.r_[rng.integers(0, n, 4000), np.full(n, n - 1), np.arange(n)]
ib = np.r_[rng.integers(0, n, 4000), np.arange(n), np.full(n, n - 1)]
want = O.pairs_idx(O.pairs_f32, {"edr": 1, "lcss": 2}[m], pts, off, lens, ia, ib, eps=3e-2)[1]
assert np.array_equal(cnt.cpu().numpy()[ia, ib], want)
print("EQUAL")
"""


@pytest.mark.parametrize("measure", ["edr", "lcss"])
@pytest.mark.parametrize("n,longest", [(9, 1100), (1000, 500), (2000, 280)])
def test_counts_between_the_two_limits(measure, n, longest):
    r = subprocess.run([sys.executable, "-c", COUNTS, measure, str(n), str(longest)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "EQUAL" in r.stdout, r.stderr
